// Routing of a mixture-of-experts feed-forward.
//
// router_topk: logits z = x W_r^T (+ bias) arrive in fp32 [T, E]; the `top` largest are chosen (the
//   lower index wins a tie) and their weights are the softmax over the chosen logits only.  Written as
//   a dense map wt [T, E] (zero for experts not chosen) and as lists idx / w [T, top].
// router_grouped: the logits cover N = E + I outputs, the last I of which stand for experts that return their
//   input.  Scores s = softmax(z) over all N; the choice is made on s + correction: the N outputs form `groups`
//   equal runs of neighbours, a group's score is its largest choice score, only members of the `keep` best groups
//   can be chosen (the others count as minus infinity), and of those the `top` largest are (the lower index wins a
//   tie everywhere).  The weights are the chosen s divided by their sum (+ 1e-20).  Written as a dense map
//   wt [T, E] over the experts with tensors, as wid [T] (the sum of the weights of chosen identity experts) and
//   as lists idx / w [T, top].
// moe_scale: act[t, e*F + i] *= wt[t, e] for the E routed experts' blocks of F activations; columns
//   beyond E*F (an expert that every token uses) are left as they are.
//
// Prompts run the experts' products over the tokens that chose them (gemm_tc.cu, grouped launches):
// moe_sort: the (token, choice) pairs of a step by expert, in one block: counts, offsets, places.  An expert's rows follow one
//   another without gaps; `groups` lists its row tiles of 128.
// moe_gather: xs[row] = x[row_token[row]] (16-byte copies).
// moe_combine: residual[t, :] += the sum over t's choices of y[pos] (choices in order, so the order of the additions is fixed).
#include "common.cuh"

using namespace iert;

namespace {

constexpr int MAX_TOP = 32;

// The routing of token t by one warp from its logits (output e at row[e * lde]).
__device__ __forceinline__ void topk_token(const float* __restrict__ row, long long lde, const float* __restrict__ bias, int E, int top,
                                           float* __restrict__ wt, int ldw, int* __restrict__ idx, float* __restrict__ w, int t, int lane) {
  int chosen[MAX_TOP];
  float val[MAX_TOP];
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      bool taken = false;
      for (int j = 0; j < k; ++j) taken |= chosen[j] == e;
      const float v = row[e * lde] + (bias ? bias[e] : 0.f);
      if (!taken && (v > best || (v == best && e < bi))) { best = v; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    chosen[k] = bi;
    val[k] = best;
  }
  float den = 0.f;
  const float largest = val[0];
  for (int k = 0; k < top; ++k) { val[k] = expf(val[k] - largest); den += val[k]; }
  for (int e = lane; e < ldw; e += 32) wt[(size_t)t * ldw + e] = e < E ? 0.f : 1.f;      // (what every token uses has weight 1)
  __syncwarp();
  if (lane == 0)
    for (int k = 0; k < top; ++k) {
      const float p = val[k] / den;
      if (chosen[k] < E) wt[(size_t)t * ldw + chosen[k]] = p;
      idx[(size_t)t * top + k] = chosen[k];
      w[(size_t)t * top + k] = p;
    }
}

__global__ void router_topk_kernel(const float* __restrict__ z, long long ldz, long long lde, const float* __restrict__ bias,
                                   int E, int top, float* __restrict__ wt, int ldw, int* __restrict__ idx,
                                   float* __restrict__ w) {
  // one warp per token
  pdl_launch_dependents();     // the next kernel may start its preamble now
  pdl_wait();                  // everything below may depend on the kernel before
  topk_token(z + (size_t)blockIdx.x * ldz, lde, bias, E, top, wt, ldw, idx, w, blockIdx.x, threadIdx.x);
}

// A block per token, whose first warp routes; shared memory: s[N], c[N], group score [groups], flags [N] (bytes).  Output e of token t is
// z[t * ldz + e * lde]: rows of tokens (lde = 1) or rows of outputs (ldz = 1).
//   score_mode   0: scores are the softmax over all N outputs; 1: every output's own sigmoid
//   group_mode   0: a group's score is its best choice score; 1: the sum of its two best (of its one, if it has one)
//   weights      chosen scores / (their sum + weight_eps) * weight_scale; with renorm 0 chosen scores * weight_scale
//   ldw          row stride of wt; with shared_gate the output behind the last (number N) is the logit of a gate on an expert
//                every token uses: wt[t, E] = sigmoid(z[N]) (ldw > E)
//   x, residual  (optional) the identity experts' share is added here: residual[t] += wid[t] * x[t], by all the block's warps
struct RouterArgs {
  const float* z;
  long long ldz, lde;
  const float* correction;
  int E, N, top, groups, keep, score_mode, group_mode;
  float weight_eps, weight_scale;
  int renorm, shared_gate, ldw;
  float* wt;
  float* wid;
  int* idx;
  float* w;
};

// The routing of token t by one warp; returns the identity experts' share (in lane 0).
__device__ __forceinline__ float route_token(const RouterArgs& a, int t, int lane, float* rsm) {
  const int E = a.E, N = a.N, top = a.top, groups = a.groups, keep = a.keep;
  const long long lde = a.lde;
  float* s = rsm;
  float* c = rsm + N;
  float* gs = rsm + 2 * N;
  unsigned char* open = reinterpret_cast<unsigned char*>(rsm + 2 * N + groups);      // 1: may still be chosen
  const int per = N / groups;
  const float* row = a.z + (size_t)t * a.ldz;
  const float* correction = a.correction;
  float den = 1.f;
  if (a.score_mode == 0) {
    float m = -INFINITY;
    for (int e = lane; e < N; e += 32) m = fmaxf(m, row[e * lde]);
    m = warp_max(m);
    den = 0.f;
    for (int e = lane; e < N; e += 32) { const float p = expf(row[e * lde] - m); s[e] = p; den += p; }
    den = warp_sum(den);
  } else {
    for (int e = lane; e < N; e += 32) s[e] = 1.0f / (1.0f + expf(-row[e * lde]));
  }
  for (int e = lane; e < N; e += 32) {
    s[e] = s[e] / den;
    c[e] = s[e] + (correction ? correction[e] : 0.f);
    open[e] = 0;
  }
  __syncwarp();
  for (int g = lane; g < groups; g += 32) {
    float best = -INFINITY, second = -INFINITY;
    for (int j = 0; j < per; ++j) {
      const float v = c[g * per + j];
      if (v > best) { second = best; best = v; }
      else if (v > second) second = v;
    }
    gs[g] = a.group_mode == 1 && per > 1 ? best + second : best;
  }
  __syncwarp();
  // the `keep` best groups, one after the other; a group that was taken is marked by NaN
  for (int k = 0; k < keep; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int g = lane; g < groups; g += 32) {
      const float v = gs[g];
      if (v == v && (v > best || (v == best && g < bi) || bi == 0x7fffffff)) { best = v; bi = g; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > best || (ov == best && oi < bi))) { best = ov; bi = oi; }
    }
    __syncwarp();
    if (bi != 0x7fffffff) {
      for (int j = lane; j < per; j += 32) open[bi * per + j] = 1;
      if (lane == 0) gs[bi] = __int_as_float(0x7fc00000);
    }
    __syncwarp();
  }
  int chosen[MAX_TOP];
  float val[MAX_TOP];
  float sum = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < N; e += 32) {
      const float v = c[e];
      if (open[e] && (bi == 0x7fffffff || v > best || (v == best && e < bi))) { best = v; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > best || (ov == best && oi < bi))) { best = ov; bi = oi; }
    }
    __syncwarp();
    chosen[k] = bi;
    val[k] = bi != 0x7fffffff ? s[bi] : 0.f;
    sum += val[k];
    if (lane == 0 && bi != 0x7fffffff) open[bi] = 0;
    __syncwarp();
  }
  float* wt = a.wt + (size_t)t * a.ldw;
  for (int e = lane; e < E; e += 32) wt[e] = 0.f;
  __syncwarp();
  float identity = 0.f;
  if (lane == 0) {
    for (int k = 0; k < top; ++k) {
      const float p = a.renorm ? val[k] / (sum + a.weight_eps) * a.weight_scale : val[k] * a.weight_scale;
      if (chosen[k] < E) wt[chosen[k]] = p;
      else if (chosen[k] < N) identity += p;
      a.idx[(size_t)t * top + k] = chosen[k] < N ? chosen[k] : -1;
      a.w[(size_t)t * top + k] = p;
    }
    a.wid[t] = identity;
    if (a.shared_gate) wt[E] = 1.0f / (1.0f + expf(-row[N * lde]));
  }
  return identity;
}

template <typename TX>
__global__ void router_grouped_kernel(RouterArgs a, const TX* __restrict__ x, long long ldx, float* __restrict__ residual, long long ldres, int H) {
  extern __shared__ float rsm[];
  __shared__ float share_s;
  pdl_launch_dependents();     // the next kernel (the experts' product) may fetch its first weights now
  pdl_wait();
  const int t = blockIdx.x;
  if (threadIdx.x < 32) {
    const float share = route_token(a, t, threadIdx.x, rsm);
    if (threadIdx.x == 0) share_s = share;
  }
  if (!x) return;
  __syncthreads();
  const float share = share_s;
  if (share == 0.f) return;
  float* out = residual + (size_t)t * ldres;
  const TX* in = x + (size_t)t * ldx;
  if (H % 4 == 0 && ldx % 4 == 0 && ldres % 4 == 0 && (((uintptr_t)residual | (uintptr_t)x) & 15) == 0) {
    for (int i = threadIdx.x * 4; i < H; i += blockDim.x * 4) {
      float4 o = *reinterpret_cast<const float4*>(out + i);
      float v[4];
      if (sizeof(TX) == 2) {
        const uint2 raw = *reinterpret_cast<const uint2*>(in + i);
        const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        v[0] = f0.x; v[1] = f0.y; v[2] = f1.x; v[3] = f1.y;
      } else {
        const float4 f = *reinterpret_cast<const float4*>(in + i);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      }
      o.x += share * v[0]; o.y += share * v[1]; o.z += share * v[2]; o.w += share * v[3];
      *reinterpret_cast<float4*>(out + i) = o;
    }
    return;
  }
  for (int i = threadIdx.x; i < H; i += blockDim.x) out[i] += share * to_f32(in[i]);
}

template <typename T>
__global__ void moe_scale_kernel(T* __restrict__ act, long long ld, const float* __restrict__ wt, int ldw, int E, int F) {
  pdl_launch_dependents();     // the down product may fetch its first weights now
  pdl_wait();
  const int t = blockIdx.x;
  T* row = act + (size_t)t * ld;
  if (sizeof(T) == 2 && F % 8 == 0 && ld % 8 == 0 && ((uintptr_t)act & 15) == 0) {      // eight at a time
    for (int i = threadIdx.x * 8; i < E * F; i += blockDim.x * 8) {
      const float w = wt[(size_t)t * ldw + i / F];
      uint4 v = *reinterpret_cast<const uint4*>(row + i);
      __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(p[e]);
        p[e] = __floats2bfloat162_rn(f.x * w, f.y * w);
      }
      *reinterpret_cast<uint4*>(row + i) = v;
    }
    return;
  }
  for (int i = threadIdx.x; i < E * F; i += blockDim.x)
    row[i] = from_f32<T>(to_f32(row[i]) * wt[(size_t)t * ldw + i / F]);
}

// One-token steps: the router's product and the routing in one kernel, a block per token.  A warp takes every eighth output, a lane
// eight numbers of the row at a time; fp32 sums.  The tensor-core product has one tile of up to 32 columns to give to 148 SMs, splits it
// over k and adds the parts through memory: 20 us and 8 more for the routing at 32 tokens x 16 outputs x 4,096; this kernel 16.
// GROUPED: route_token with `a`, else topk_token with the fields of `a` it needs (`correction` is the bias then).
constexpr int ROUTER_THREADS = 256;

template <bool GROUPED>
__global__ void __launch_bounds__(ROUTER_THREADS)
router_step_kernel(RouterArgs a, const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ w_r, long long ldr, int K,
                   int rows, float* __restrict__ residual, long long ldres, int H) {
  extern __shared__ float rsm[];
  __shared__ float share_s;
  float* z_s = rsm;                        // [rows] logits, then the routing's own
  pdl_launch_dependents();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const __nv_bfloat16* xr = x + (size_t)t * ldx;
  for (size_t i = (size_t)threadIdx.x * 64; t == 0 && i < (size_t)rows * K; i += ROUTER_THREADS * 64)      // (weights: ahead of the wait)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(w_r + i / K * ldr + i % K));
  pdl_wait();
  for (int e = warp; e < rows; e += 2 * (ROUTER_THREADS / 32)) {
    const int e2 = e + ROUTER_THREADS / 32;
    const __nv_bfloat16* w0 = w_r + (size_t)e * ldr;
    const __nv_bfloat16* w1 = w_r + (size_t)(e2 < rows ? e2 : e) * ldr;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
    for (int k = lane * 8; k < K; k += 256) {
      const uint4 xv = *reinterpret_cast<const uint4*>(xr + k), u = *reinterpret_cast<const uint4*>(w0 + k), v = *reinterpret_cast<const uint4*>(w1 + k);
      const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&xv);
      const __nv_bfloat162* up = reinterpret_cast<const __nv_bfloat162*>(&u);
      const __nv_bfloat162* vp = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 xf = __bfloat1622float2(xp[i]), uf = __bfloat1622float2(up[i]), vf = __bfloat1622float2(vp[i]);
        s0 = fmaf(xf.x, uf.x, s0); s0 = fmaf(xf.y, uf.y, s0);
        s1 = fmaf(xf.x, vf.x, s1); s1 = fmaf(xf.y, vf.y, s1);
      }
    }
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if (lane == 0) {
      z_s[e] = s0;
      if (e2 < rows) z_s[e2] = s1;
    }
  }
  __syncthreads();
  if (warp == 0) {
    if (GROUPED) {
      a.z = z_s;
      a.ldz = 0;
      a.lde = 1;
      const float share = route_token(a, t, lane, rsm + rows);
      if (lane == 0) share_s = share;
    } else {
      topk_token(z_s, 1, a.correction, a.E, a.top, a.wt, a.ldw, a.idx, a.w, t, lane);
    }
  }
  if (!GROUPED || !residual) return;
  __syncthreads();
  const float share = share_s;
  if (share == 0.f) return;
  for (int i = threadIdx.x; i < H; i += ROUTER_THREADS) residual[(size_t)t * ldres + i] += share * __bfloat162float(xr[i]);
}

constexpr int SORT_THREADS = 1024, ROW_TILE = 128;

__global__ void __launch_bounds__(SORT_THREADS)
moe_sort_kernel(const int* __restrict__ idx, const float* __restrict__ w, int pairs, int top, int E, int* __restrict__ groups,
                int* __restrict__ pos, int* __restrict__ row_token, float* __restrict__ row_w) {
  extern __shared__ int sm_sort[];
  int* count = sm_sort;                  // [E]
  int* next = sm_sort + E;               // [E] the expert's next free row
  int* tile0 = sm_sort + 2 * E;          // [E] its first row tile
  pdl_launch_dependents();
  for (int e = threadIdx.x; e < E; e += SORT_THREADS) count[e] = 0;
  __syncthreads();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int rounds = (pairs + SORT_THREADS - 1) / SORT_THREADS;
  auto expert_of = [&](int i) {
    const int e = i < pairs ? idx[i] : -1;
    return e >= 0 && e < E ? e : -1;     // experts without tensors, and choices that could not be made, have no rows
  };
  for (int r = 0; r < rounds; ++r) {
    const int e = expert_of(r * SORT_THREADS + threadIdx.x);
    const unsigned same = __match_any_sync(0xffffffffu, e);
    if (e >= 0 && lane == __ffs(same) - 1) atomicAdd(&count[e], __popc(same));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int rows = 0, tiles = 0;
    for (int e = 0; e < E; ++e) {
      next[e] = rows;
      tile0[e] = tiles;
      rows += count[e];
      tiles += (count[e] + ROW_TILE - 1) / ROW_TILE;
    }
    groups[0] = tiles;
    groups[1] = rows;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += SORT_THREADS)
    for (int t = 0; t * ROW_TILE < count[e]; ++t) {
      int* g = groups + 2 + 3 * (tile0[e] + t);
      g[0] = e;
      g[1] = next[e] + t * ROW_TILE;
      g[2] = next[e] + count[e];
    }
  __syncthreads();
  for (int r = 0; r < rounds; ++r) {
    const int i = r * SORT_THREADS + threadIdx.x;
    const int e = expert_of(i);
    const unsigned same = __match_any_sync(0xffffffffu, e);
    int row = 0;
    if (e >= 0 && lane == __ffs(same) - 1) row = atomicAdd(&next[e], __popc(same));
    row = __shfl_sync(0xffffffffu, row, __ffs(same) - 1) + __popc(same & ((1u << lane) - 1u));
    if (i < pairs) pos[i] = e >= 0 ? row : -1;
    if (e >= 0) { row_token[row] = i / top; row_w[row] = w[i]; }
  }
}

__global__ void __launch_bounds__(256) moe_gather_kernel(const uint4* __restrict__ x, long long ldx16, const int* __restrict__ groups,
                                                         const int* __restrict__ row_token, uint4* __restrict__ xs, int width16) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x;
  if (row >= groups[1]) return;
  const uint4* src = x + (size_t)row_token[row] * ldx16;
  uint4* dst = xs + (size_t)row * width16;
  for (int i = threadIdx.x; i < width16; i += 4 * 256) {
    uint4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) if (i + k * 256 < width16) v[k] = src[i + k * 256];
#pragma unroll
    for (int k = 0; k < 4; ++k) if (i + k * 256 < width16) dst[i + k * 256] = v[k];
  }
}

__global__ void __launch_bounds__(256) moe_combine_kernel(const float* __restrict__ y, const int* __restrict__ pos, const float* __restrict__ w,
                                                          int top, float* __restrict__ residual, long long ldres, int H) {
  __shared__ int pos_s[MAX_TOP];
  __shared__ float w_s[MAX_TOP];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  if (threadIdx.x < top) {
    pos_s[threadIdx.x] = pos[(size_t)t * top + threadIdx.x];
    w_s[threadIdx.x] = w[(size_t)t * top + threadIdx.x];
  }
  __syncthreads();
  for (int i = threadIdx.x * 4; i < H; i += 256 * 4) {
    float4* out = reinterpret_cast<float4*>(residual + (size_t)t * ldres + i);
    float4 o = *out, a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < top; ++k) {
      if (pos_s[k] < 0) {                // no rows: an expert without tensors, or no choice for want of a number
        const float n = w_s[k] != w_s[k] ? w_s[k] : 0.f;
        a.x += n; a.y += n; a.z += n; a.w += n;
        continue;
      }
      const float4 v = *reinterpret_cast<const float4*>(y + (size_t)pos_s[k] * H + i);
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
    o.x += a.x; o.y += a.y; o.z += a.z; o.w += a.w;
    *out = o;
  }
}

}  // namespace

// idx, w [n_tokens, top] as the routers leave them.  groups: [2 + 3 * (n_tokens * top / 128 + E)] ints; pos [n_tokens * top];
// row_token, row_w [n_tokens * top].
IERT_API int iert_moe_sort(const int* idx, const float* w, int n_tokens, int top, int E, int* groups, int* pos, int* row_token,
                           float* row_w, cudaStream_t stream) {
  if (n_tokens <= 0) return IERT_OK;
  if (top <= 0 || E <= 0 || E > 1024 || (long long)n_tokens * top > (1 << 24)) return IERT_BAD_ARGUMENT;
  launch_dep(moe_sort_kernel, dim3(1), dim3(SORT_THREADS), 3 * E * sizeof(int), stream, idx, w, n_tokens * top, top, E, groups, pos,
             row_token, row_w);
  return iert_check_launch("moe_sort");
}

// x [*, width] bf16 with row stride ldx, xs [rows, width] bf16 (width and ldx multiples of 8, rows on 16-byte boundaries).
IERT_API int iert_moe_gather(const void* x, long long ldx, const int* groups, const int* row_token, int max_rows, void* xs, int width,
                             cudaStream_t stream) {
  if (max_rows <= 0) return IERT_OK;
  if (width <= 0 || width % 8 || ldx % 8 || (((uintptr_t)x | (uintptr_t)xs) & 15)) return IERT_BAD_ARGUMENT;
  launch_dep(moe_gather_kernel, dim3(max_rows), dim3(256), 0, stream, (const uint4*)x, ldx / 8, groups, row_token, (uint4*)xs, width / 8);
  return iert_check_launch("moe_gather");
}

// y fp32 [rows, H]; residual fp32 [n_tokens, H] with row stride ldres (H and ldres multiples of 4, rows on 16-byte boundaries).
IERT_API int iert_moe_combine(const float* y, const int* pos, const float* w, int n_tokens, int top, float* residual, long long ldres,
                              int H, cudaStream_t stream) {
  if (n_tokens <= 0) return IERT_OK;
  if (top <= 0 || top > MAX_TOP || H <= 0 || H % 4 || ldres % 4 || (((uintptr_t)y | (uintptr_t)residual) & 15)) return IERT_BAD_ARGUMENT;
  launch_dep(moe_combine_kernel, dim3(n_tokens), dim3(256), 0, stream, y, pos, w, top, residual, ldres, H);
  return iert_check_launch("moe_combine");
}

// z: output e of token t at z[t * ldz + e * lde]; wt: row stride ldw >= E, columns from E on are set to 1.
IERT_API int iert_router_topk(const float* z, long long ldz, long long lde, const float* bias, int n_tokens, int E, int top,
                              float* wt, int ldw, int* idx, float* w, cudaStream_t stream) {
  if (n_tokens <= 0) return IERT_OK;
  if (E <= 0 || top <= 0 || top > E || top > MAX_TOP || ldw < E) return IERT_BAD_ARGUMENT;
  launch_dep(router_topk_kernel, dim3(n_tokens), dim3(32), 0, stream, z, ldz, lde, bias, E, top, wt, ldw, idx, w);
  return iert_check_launch("router_topk");
}

// z: output e of token t at z[t * ldz + e * lde] (fp32).  x (optional, [n_tokens, H] of x_dtype) with residual (fp32 [n_tokens, H]): the
// identity experts' share is added there.
IERT_API int iert_router_grouped(const float* z, long long ldz, long long lde, const float* correction, int n_tokens, int E, int N, int top,
                                 int groups, int keep, int score_mode, int group_mode, float weight_eps, float weight_scale,
                                 int renorm, int shared_gate, float* wt, int ldw, float* wid, int* idx, float* w, const void* x,
                                 int x_dtype, long long ldx, float* residual, long long ldres, int H, cudaStream_t stream) {
  if (n_tokens <= 0) return IERT_OK;
  if (score_mode < 0 || score_mode > 1 || group_mode < 0 || group_mode > 1) return IERT_BAD_ARGUMENT;
  if (ldw < E + (shared_gate ? 1 : 0) || (x && (!residual || H <= 0 || (x_dtype != IERT_F32 && x_dtype != IERT_BF16)))) return IERT_BAD_ARGUMENT;
  if (E < 0 || N < E || N <= 0 || top <= 0 || top > MAX_TOP || groups <= 0 || N % groups || keep <= 0 || keep > groups ||
      top > keep * (N / groups))
    return IERT_BAD_ARGUMENT;
  const size_t smem = (size_t)(2 * N + groups) * sizeof(float) + (size_t)N;
  if (smem > 48 * 1024) return IERT_BAD_ARGUMENT;
  const RouterArgs a = {z, ldz, lde, correction, E, N, top, groups, keep, score_mode, group_mode, weight_eps, weight_scale, renorm,
                        shared_gate, ldw, wt, wid, idx, w};
  const dim3 threads(x ? 256 : 32);
  if (x && x_dtype == IERT_F32)
    launch_dep(router_grouped_kernel<float>, dim3(n_tokens), threads, smem, stream, a, (const float*)x, ldx, residual, ldres, H);
  else
    launch_dep(router_grouped_kernel<__nv_bfloat16>, dim3(n_tokens), threads, smem, stream, a, (const __nv_bfloat16*)x, ldx, residual, ldres, H);
  return iert_check_launch("router_grouped");
}

IERT_API int iert_moe_scale(void* act, int dtype, long long ld, const float* wt, int ldw, int n_tokens, int E, int F, cudaStream_t stream) {
  if (n_tokens <= 0) return IERT_OK;
  if (E < 0 || F <= 0 || ldw < E) return IERT_BAD_ARGUMENT;
  if (dtype == IERT_F32)
    launch_dep(moe_scale_kernel<float>, dim3(n_tokens), dim3(256), 0, stream, (float*)act, ld, wt, ldw, E, F);
  else if (dtype == IERT_BF16)
    launch_dep(moe_scale_kernel<__nv_bfloat16>, dim3(n_tokens), dim3(256), 0, stream, (__nv_bfloat16*)act, ld, wt, ldw, E, F);
  else return IERT_BAD_ARGUMENT;
  return iert_check_launch("moe_scale");
}

// The product of x [n_tokens, K] with the router's `rows` rows w_r (bf16) and the routing, in one kernel.  grouped != 0: as
// iert_router_grouped with weights renormalised and no shared gate (rows = N), `residual` (optional, fp32 [n_tokens, K]) receives the identity experts'
// share; else as iert_router_topk (`correction` is the bias, rows = E = N).  K and the strides multiples of 8, rows on 16-byte boundaries.
IERT_API int iert_router_step(const void* x, long long ldx, const void* w_r, long long ldr, int K, int rows, int grouped, const float* correction,
                              int n_tokens, int E, int N, int top, int groups, int keep, int score_mode, int group_mode, float weight_eps,
                              float weight_scale, float* wt, int ldw, float* wid, int* idx, float* w, float* residual, long long ldres, cudaStream_t stream) {
  if (n_tokens <= 0) return IERT_OK;
  if (K <= 0 || K % 8 || ldx % 8 || ldr % 8 || (((uintptr_t)x | (uintptr_t)w_r) & 15) || E <= 0 || N < E || top <= 0 || top > MAX_TOP)
    return IERT_BAD_ARGUMENT;
  if (grouped ? (score_mode < 0 || score_mode > 1 || group_mode < 0 || group_mode > 1 || groups <= 0 || N % groups || keep <= 0 || keep > groups ||
                 top > keep * (N / groups) || ldw < E || rows != N || !wid)
              : (top > E || ldw < E || rows != E || residual))
    return IERT_BAD_ARGUMENT;
  const size_t smem = (size_t)(rows + 2 * N + groups) * sizeof(float) + (size_t)N;
  if (smem > 47 * 1024) return IERT_BAD_ARGUMENT;
  const RouterArgs a = {nullptr, 0, 1, correction, E, N, top, groups, keep, score_mode, group_mode, weight_eps, weight_scale, 1,
                        0, ldw, wt, wid, idx, w};
  if (grouped)
    launch_dep(router_step_kernel<true>, dim3(n_tokens), dim3(ROUTER_THREADS), smem, stream, a, (const __nv_bfloat16*)x, ldx,
               (const __nv_bfloat16*)w_r, ldr, K, rows, residual, ldres, K);
  else
    launch_dep(router_step_kernel<false>, dim3(n_tokens), dim3(ROUTER_THREADS), smem, stream, a, (const __nv_bfloat16*)x, ldx,
               (const __nv_bfloat16*)w_r, ldr, K, rows, (float*)nullptr, 0, K);
  return iert_check_launch("router_step");
}
