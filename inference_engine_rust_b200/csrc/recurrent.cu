// Recurrences with a matrix state per head, S [DIM x V] in fp32, carried from token to token in the
// sequence's state.  Compiled per key size (-DDIM=...), like the attention kernels per head size.
//
// Work split: a column j of S never meets another column, so a CTA owns (sequence, head, a run of
// columns) and a thread owns RPT = ceil(DIM / R) rows of one column in registers (rows r, r + R, ...: the
// lanes of a column read neighbouring words of a token's k and q, so shared memory serves them without bank
// conflicts); the R threads of a column are neighbouring lanes and add their partial dot products by shuffles.  R is chosen at the
// launch: the tokens of a sequence are a chain, so all the parallelism there is lies in heads x columns x
// R, and a single prompt wants many lanes per column (more warps per SM to hide the chain's latency)
// where a batch of sequences is served best by few (fewer shuffles and shared-memory reads per FMA).
// A CTA walks its sequence's tokens in order; the tokens' vectors come through shared memory CHUNK
// tokens at a time, fetched (and converted) by two warps that do nothing else into the buffer the
// computing warps are not reading, so that those never wait for memory: one barrier per chunk.
// State is read when the CTA starts and written back when it ends, so a step of one token and a
// prompt of thousands run the same code.
//
//   gated delta rule, per token:   S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
//   mLSTM, per token:  m' = max(f + m, i);  S <- e^(f+m-m') S + e^(i-m') k v^T;  n likewise with k;
//                      o = S^T q / (max(|n . q|, e^(-m')) + 1e-6),  m starts at 0
//       with i = cap tanh((zi + bi) / cap),  f = logsigmoid(cap tanh((zf + bf) / cap))
//   wkv (decay per key channel, a bonus for the current token), per token:
//                      o = (S + diag(u) k v^T)^T r;  S <- diag(w) S + k v^T
#include "common.cuh"

#include <stdlib.h>

using namespace iert;

#ifndef DIM
#error "compile with -DDIM=<rows of the state matrix>"
#endif

namespace {

constexpr int fewest_lanes() {                 // the fewest lanes per column that keep a thread's rows at 32 or fewer
  int r = 1;
  while ((DIM + r - 1) / r > 32 && r < 32) r *= 2;
  return r;
}
constexpr int R_MIN = fewest_lanes();
constexpr int CHUNK = DIM <= 128 ? 8 : DIM <= 256 ? 4 : DIM <= 512 ? 2 : 1;
constexpr int LOADERS = 64;                    // threads of a CTA that only fetch

template <int R>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = R / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct DeltaArgs {
  const float* qkv;      // [T, C] fp32: q [G*DIM] | k [G*DIM] | v [H*V]   (from delta_prep)
  const float* beta;     // [T, H]
  const float* decay;    // [T, H]
  float* state;          // per slot at s_off: S [H, DIM, V]
  long long state_stride, s_off;
  float* o;              // [T, H*V] fp32
  int G, H, V, cols;
};

template <int R>
__global__ void __launch_bounds__(256 + LOADERS) delta_recur_kernel(DeltaArgs a, IertBatchView b) {
  constexpr int RPT = (DIM + R - 1) / R;
  __shared__ __align__(16) float k_s[2][CHUNK][DIM], q_s[2][CHUNK][DIM], v_s[2][CHUNK][256], bg_s[2][CHUNK][2];
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * a.cols;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const int workers = blockDim.x - LOADERS;
  const bool loader = (int)threadIdx.x >= workers;
  const int col = threadIdx.x / R, r = threadIdx.x % R;
  const int j = c0 + col;
  const bool live = !loader && col < a.cols && j < a.V;
  const int g = head / (a.H / a.G);
  const int GD = a.G * DIM, C = 2 * GD + a.H * a.V;
  auto fetch = [&](int buf, int tc, int tid, int nthreads) {
    const int n = min(CHUNK, t1 - tc);
    if (DIM % 4 == 0 && C % 4 == 0 && ((uintptr_t)a.qkv & 15) == 0) {       // 16-byte loads
      // every load of the chunk is issued before the first is stored (a loader's loads are all it waits for)
      constexpr int ITER = (CHUNK * (DIM / 4) + LOADERS - 1) / LOADERS > 0 ? (CHUNK * (DIM / 4) + LOADERS - 1) / LOADERS : 1;
      float4 qv[ITER], kv[ITER];
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 4)) {
          const int tt = x / (DIM / 4), d = 4 * (x - tt * (DIM / 4));
          const float* rowp = a.qkv + (size_t)(tc + tt) * C;
          qv[it] = *reinterpret_cast<const float4*>(rowp + g * DIM + d);
          kv[it] = *reinterpret_cast<const float4*>(rowp + GD + g * DIM + d);
        }
      }
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 4)) {
          const int tt = x / (DIM / 4), d = 4 * (x - tt * (DIM / 4));
          *reinterpret_cast<float4*>(&q_s[buf][tt][d]) = qv[it];
          *reinterpret_cast<float4*>(&k_s[buf][tt][d]) = kv[it];
        }
      }
    } else {
      for (int x = tid; x < n * DIM; x += nthreads) {
        const int tt = x / DIM, d = x - tt * DIM;
        const float* rowp = a.qkv + (size_t)(tc + tt) * C;
        q_s[buf][tt][d] = rowp[g * DIM + d];
        k_s[buf][tt][d] = rowp[GD + g * DIM + d];
      }
    }
    for (int x = tid; x < n * a.cols; x += nthreads) {
      const int tt = x / a.cols, cc = x - tt * a.cols;
      v_s[buf][tt][cc] = c0 + cc < a.V ? a.qkv[(size_t)(tc + tt) * C + 2 * GD + head * a.V + c0 + cc] : 0.f;
    }
    if (tid < n) {
      bg_s[buf][tid][0] = a.beta[(size_t)(tc + tid) * a.H + head];
      bg_s[buf][tid][1] = a.decay[(size_t)(tc + tid) * a.H + head];
    }
  };
  float* Sg = a.state + (size_t)slot * a.state_stride + a.s_off + (size_t)head * DIM * a.V;
  float S[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int d = i * R + r;
    S[i] = (live && d < DIM) ? Sg[(size_t)d * a.V + j] : 0.f;
  }
  fetch(0, t0, threadIdx.x, blockDim.x);
  __syncthreads();
  int buf = 0;
  for (int tc = t0; tc < t1; tc += CHUNK, buf ^= 1) {
    const int n = min(CHUNK, t1 - tc);
    if (loader) {
      if (tc + CHUNK < t1) fetch(buf ^ 1, tc + CHUNK, threadIdx.x - workers, LOADERS);
    } else {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) {
        if (tt >= n) break;
        const float beta = bg_s[buf][tt][0], gd = bg_s[buf][tt][1];
        float kk[RPT];
        float dk = 0.f;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int d = i * R + r;
          kk[i] = d < DIM ? k_s[buf][tt][d] : 0.f;
          S[i] *= gd;
          dk = fmaf(S[i], kk[i], dk);
        }
        dk = group_sum<R>(dk);
        const float u = beta * ((live ? v_s[buf][tt][col] : 0.f) - dk);
        float oq = 0.f;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int d = i * R + r;
          S[i] = fmaf(kk[i], u, S[i]);
          oq = fmaf(S[i], d < DIM ? q_s[buf][tt][d] : 0.f, oq);
        }
        oq = group_sum<R>(oq);
        if (live && r == 0) a.o[(size_t)(tc + tt) * a.H * a.V + (size_t)head * a.V + j] = oq;
      }
    }
    __syncthreads();
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int d = i * R + r;
      if (d < DIM) Sg[(size_t)d * a.V + j] = S[i];
    }
  }
}

// ---- prompts: eight tokens at a time ---------------------------------------------------------------------------------
// Token after token, a step's time is the latency of its chain (dot product, shuffles, update: about 680 cycles a token), not its
// work.  Over a chunk of c = 8 tokens with decays g and G_i = g_1 .. g_i, the state in front of the chunk S and u_i as above:
//
//   S_i = G_i S + sum_{j <= i} (G_i / G_j) k_j u_j      so      u_i = beta_i (v_i - G_i k_i.S - sum_{j < i} (G_i / G_j) (k_i.k_j) u_j)
//   o_i = G_i q_i.S + sum_{j <= i} (G_i / G_j) (q_i.k_j) u_j
//
// The sixteen dot products k_i.S, q_i.S of a column are independent: all their partial sums are formed first and then added
// over the 16 lanes of the column together, each lane ending with one of them (15 shuffles instead of 64); what is left of
// the chain is eight steps of one broadcast and one multiply-add.  The tokens' products k_i.k_j, q_i.k_j (the same for all
// columns) with the ratios (products of the decays between, never quotients) come from a kernel in front, which has a block per
// chunk and key head; a loader warp brings everything through a ring of four chunks.  Everything is fp32.
// A thread owns DIM / 16 rows of FOUR columns, so that a token's k and q, read from shared memory, serve four columns (with two
// columns and twice the warps: 448 us against 404 over 2,048 tokens, 32 heads of 128 x 128).  Two rows share an
// instruction: 344 us.
#define IERT_CHUNKED (DIM == 64 || DIM == 128)                // (larger sizes would not fit the registers)
#if IERT_CHUNKED
constexpr int CT = 8, CG = 4, CL = 16, CWORK = 128, CCOLS = CWORK / CL * CG;
constexpr int CP = DIM / CL / 2;                              // pairs of rows per lane
constexpr int RING = 4;                                       // chunks in shared memory
// per token and head: 8 coefficients of earlier u in u_i, 8 in o_i, then G_i, G_8 / G_i, beta_i, G_8
constexpr int COEF = 20;

// A lane's rows 64 x + 4 r .. + 3 of a vector in shared memory.
__device__ __forceinline__ void own_rows(float2 (&v)[CP], const float* src, int r) {
#pragma unroll
  for (int x = 0; x < CP / 2; ++x) {
    const float4 f = *reinterpret_cast<const float4*>(src + 64 * x + 4 * r);
    v[2 * x] = make_float2(f.x, f.y);
    v[2 * x + 1] = make_float2(f.z, f.w);
  }
}
// The rows 64 x + 4 r .. + 3 of four columns of the state, from memory and back.
__device__ __forceinline__ void load_rows(float2 (&S)[CP][CG], const float* Sg, int V, int r, bool live) {
#pragma unroll
  for (int i = 0; i < CP; ++i) {
    const float* p = Sg + (size_t)((i / 2) * 64 + 4 * r + (i % 2) * 2) * V;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 u = live ? *reinterpret_cast<const float4*>(p) : z, v = live ? *reinterpret_cast<const float4*>(p + V) : z;
    S[i][0] = make_float2(u.x, v.x); S[i][1] = make_float2(u.y, v.y); S[i][2] = make_float2(u.z, v.z); S[i][3] = make_float2(u.w, v.w);
  }
}
__device__ __forceinline__ void store_rows(const float2 (&S)[CP][CG], float* Sg, int V, int r) {
#pragma unroll
  for (int i = 0; i < CP; ++i) {
    float* p = Sg + (size_t)((i / 2) * 64 + 4 * r + (i % 2) * 2) * V;
    *reinterpret_cast<float4*>(p) = make_float4(S[i][0].x, S[i][1].x, S[i][2].x, S[i][3].x);
    *reinterpret_cast<float4*>(p + V) = make_float4(S[i][0].y, S[i][1].y, S[i][2].y, S[i][3].y);
  }
}

__device__ __forceinline__ void copy16(void* dst, const void* src, bool in) {      // zeros where there is nothing to read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// The chunk that block `x` of a grid over all sequences' chunks looks after: first token and end of the sequence; false: none.
__device__ __forceinline__ bool chunk_of(const IertBatchView& b, int x, int& tc, int& t1) {
  for (int s = 0; s < b.n_seqs; ++s) {
    const int lo = b.cu_q[s], hi = b.cu_q[s + 1], n = (hi - lo + CT - 1) / CT;
    if (x < n) {
      tc = lo + x * CT;
      t1 = hi;
      return b.slot_ids[s] >= 0;
    }
    x -= n;
  }
  return false;
}

// Block (chunk, key head): a thread per product of two of the chunk's tokens, then per coefficient of each head that shares them.
// (No early start for the kernel behind: its blocks want an SM each, and would be packed in pairs beside this kernel's.)
__global__ void __launch_bounds__(128) delta_coef_kernel(DeltaArgs a, float* __restrict__ coef, IertBatchView b) {
  __shared__ __align__(16) float k_s[CT][DIM + 4], q_s[CT][DIM + 4];
  __shared__ float dot_s[2 * CT][CT], g_s[CT], beta_s[CT];
  pdl_wait();
  int tc, t1;
  if (!chunk_of(b, blockIdx.x, tc, t1)) return;
  const int g = blockIdx.y, GD = a.G * DIM, C = 2 * GD + a.H * a.V, n = min(CT, t1 - tc), rep = a.H / a.G;
  for (int x = threadIdx.x; x < CT * DIM / 4; x += 128) {
    const int t = x / (DIM / 4), d = 4 * (x % (DIM / 4));
    const float* row = a.qkv + (size_t)(tc + min(t, n - 1)) * C + g * DIM + d;
    *reinterpret_cast<float4*>(&q_s[t][d]) = *reinterpret_cast<const float4*>(row);
    *reinterpret_cast<float4*>(&k_s[t][d]) = *reinterpret_cast<const float4*>(row + GD);
  }
  __syncthreads();
  const int row = threadIdx.x / CT, j = threadIdx.x % CT, i = row % CT;      // row i of u, or row 8 + i of o
  const bool used = j < i + (row >= CT ? 1 : 0);
  if (used) {
    const float* x = row < CT ? k_s[i] : q_s[i];
    const float* y = k_s[j];
    float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll 8
    for (int d = 0; d < DIM; d += 4) {
      const float4 u = *reinterpret_cast<const float4*>(x + d), v = *reinterpret_cast<const float4*>(y + d);
      d0 = fmaf(u.x, v.x, d0); d1 = fmaf(u.y, v.y, d1); d2 = fmaf(u.z, v.z, d2); d3 = fmaf(u.w, v.w, d3);
    }
    dot_s[row][j] = (d0 + d1) + (d2 + d3);
  }
  for (int h = g * rep; h < (g + 1) * rep; ++h) {
    __syncthreads();
    if (threadIdx.x < CT) {
      const bool in = (int)threadIdx.x < n;
      beta_s[threadIdx.x] = in ? a.beta[(size_t)(tc + threadIdx.x) * a.H + h] : 0.f;
      g_s[threadIdx.x] = in ? a.decay[(size_t)(tc + threadIdx.x) * a.H + h] : 1.f;
    }
    __syncthreads();
    if (i < n) {
      float* out = coef + ((size_t)(tc + i) * a.H + h) * COEF;
      float ratio = 1.f;
      for (int m = j + 1; m <= i; ++m) ratio *= g_s[m];
      const float v = used ? dot_s[row][j] * ratio : 0.f;
      out[(row >= CT ? CT : 0) + j] = row < CT ? -beta_s[i] * v : v;
      if (row < CT && j < 4) {
        float to = 1.f, from = 1.f;
        for (int m = 0; m <= i; ++m) to *= g_s[m];
        for (int m = i + 1; m < CT; ++m) from *= g_s[m];
        out[2 * CT + j] = j == 0 ? to : j == 1 ? from : j == 2 ? beta_s[i] : to * from;
      }
    }
  }
}

// Sum over the 16 lanes of a column of 2 * HALF values per column: the lanes whose bit MASK is set keep the upper half.
template <int HALF, int MASK>
__device__ __forceinline__ void halve(float (&v)[16][CG], bool upper) {
#pragma unroll
  for (int m = 0; m < HALF; ++m)
#pragma unroll
    for (int c = 0; c < CG; ++c) {
      const float send = upper ? v[m][c] : v[m + HALF][c], keep = upper ? v[m + HALF][c] : v[m][c];
      v[m][c] = keep + __shfl_xor_sync(0xffffffffu, send, MASK);
    }
}

__global__ void __launch_bounds__(CWORK + 32) delta_chunk_kernel(DeltaArgs a, const float* __restrict__ coef, IertBatchView b) {
  __shared__ __align__(16) float k_s[RING][CT][DIM], q_s[RING][CT][DIM], v_s[RING][CT][CCOLS], c_s[RING][CT][COEF];
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * CCOLS;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const int n_chunks = (t1 - t0 + CT - 1) / CT;

  if (threadIdx.x >= CWORK) {
    // ---------------- loader: one warp, three chunks ahead ----------------
    const int lane = threadIdx.x - CWORK, g = head / (a.H / a.G), GD = a.G * DIM, C = 2 * GD + a.H * a.V;
    auto ask = [&](int n) {
      if (n < n_chunks) {
        const int tc = t0 + n * CT, buf = n % RING;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
          const bool in = tc + t < t1;
          const size_t tok = in ? tc + t : t0;
          const float* row = a.qkv + tok * C;
          if (lane < DIM / 4) {
            copy16(&q_s[buf][t][4 * lane], row + g * DIM + 4 * lane, in);
            copy16(&k_s[buf][t][4 * lane], row + GD + g * DIM + 4 * lane, in);
          }
          if (lane < CCOLS / 4) {
            const bool col = c0 + 4 * lane < a.V;
            copy16(&v_s[buf][t][4 * lane], row + 2 * GD + (col ? head * a.V + c0 + 4 * lane : 0), in && col);
          } else if (lane < CCOLS / 4 + COEF / 4) {
            const int x = 4 * (lane - CCOLS / 4);
            copy16(&c_s[buf][t][x], coef + (tok * a.H + head) * COEF + x, in);
          }
        }
      }
      copies_commit();
    };
    for (int n = 0; n < RING - 1; ++n) ask(n);
    copies_wait<RING - 2>();
    __syncthreads();
    for (int n = 0; n < n_chunks; ++n) {
      ask(n + RING - 1);                 // its place was read before the last barrier
      copies_wait<RING - 2>();           // chunk n + 1 has arrived
      __syncthreads();
    }
    return;
  }

  // ---------------- workers ----------------
  const int r = threadIdx.x % CL, grp = threadIdx.x / CL, j0 = c0 + grp * CG;
  const bool live = j0 < a.V;
  const int i_own = r & (CT - 1), limit = r < CT ? r : i_own + 1;
  float* Sg = a.state + (size_t)slot * a.state_stride + a.s_off + (size_t)head * DIM * a.V + j0;
  float2 S[CP][CG];
  load_rows(S, Sg, a.V, r, live);
  __syncthreads();
  for (int n = 0; n < n_chunks; ++n) {
    const int buf = n % RING;
    float2 kk[CT][CP];
    float v[16][CG];
#pragma unroll
    for (int t = 0; t < CT; ++t) {
      float2 qq[CP];
      own_rows(kk[t], k_s[buf][t], r);
      own_rows(qq, q_s[buf][t], r);
#pragma unroll
      for (int c = 0; c < CG; ++c) {
        float2 dk = make_float2(0.f, 0.f), dq = dk;
#pragma unroll
        for (int i = 0; i < CP; ++i) { dk = fma2(S[i][c], kk[t][i], dk); dq = fma2(S[i][c], qq[i], dq); }
        v[t][c] = dk.x + dk.y;
        v[CT + t][c] = dq.x + dq.y;
      }
    }
    halve<8, 8>(v, r & 8);
    halve<4, 4>(v, r & 4);
    halve<2, 2>(v, r & 2);
    halve<1, 1>(v, r & 1);               // lane r: k_r.S (r < 8) or q_(r - 8).S of the four columns
    const float4 sc = *reinterpret_cast<const float4*>(&c_s[buf][i_own][2 * CT]);
    const float G = sc.x, beta = sc.z;
    const float4 vt = *reinterpret_cast<const float4*>(&v_s[buf][i_own][grp * CG]);
    const float vv[CG] = {vt.x, vt.y, vt.z, vt.w};
    float co[CT], x[CG], u[CT][CG];
    *reinterpret_cast<float4*>(co) = *reinterpret_cast<const float4*>(&c_s[buf][i_own][r & CT]);
    *reinterpret_cast<float4*>(co + 4) = *reinterpret_cast<const float4*>(&c_s[buf][i_own][(r & CT) + 4]);
#pragma unroll
    for (int c = 0; c < CG; ++c) x[c] = r < CT ? beta * (vv[c] - G * v[0][c]) : G * v[0][c];
#pragma unroll
    for (int j = 0; j < CT; ++j)
#pragma unroll
      for (int c = 0; c < CG; ++c) {
        u[j][c] = __shfl_sync(0xffffffffu, x[c], j, CL);
        if (j < limit) x[c] = fmaf(co[j], u[j][c], x[c]);
      }
    if (live && r >= CT && t0 + n * CT + i_own < t1)
      *reinterpret_cast<float4*>(a.o + (size_t)(t0 + n * CT + i_own) * a.H * a.V + (size_t)head * a.V + j0) = make_float4(x[0], x[1], x[2], x[3]);
    const float2 G8 = make_float2(c_s[buf][0][2 * CT + 3], c_s[buf][0][2 * CT + 3]);
#pragma unroll
    for (int i = 0; i < CP; ++i)
#pragma unroll
      for (int c = 0; c < CG; ++c) S[i][c] = mul2(S[i][c], G8);
#pragma unroll
    for (int j = 0; j < CT; ++j) {
      const float f = c_s[buf][j][2 * CT + 1];
#pragma unroll
      for (int c = 0; c < CG; ++c) {
        const float2 uw = make_float2(f * u[j][c], f * u[j][c]);
#pragma unroll
        for (int i = 0; i < CP; ++i) S[i][c] = fma2(kk[j][i], uw, S[i][c]);
      }
    }
    __syncthreads();
  }
  if (live) store_rows(S, Sg, a.V, r);
}
#endif

struct MlstmArgs {
  const void* proj;      // [T, ld] run dtype: q [H*DIM] | k [H*DIM] | v [H*V] | ...
  long long ld;
  const float* gates;    // [T, gld] fp32: zi [H] | zf [H]
  long long gld;
  const float* bi;       // [H]
  const float* bf;       // [H]
  float cap;
  float* state;          // per slot: S [H, DIM, V] at s_off, n [H, DIM] at n_off, m [H] at m_off
  long long state_stride, s_off, n_off, m_off;
  float* coef;           // [T, H, 3] fp32: e^(f+m-m'), e^(i-m'), the read-out's denominator
  float* o;              // [T, H*V] fp32
  int H, V, cols;
};

__device__ __forceinline__ float logsigmoid_f(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// The part of the recurrence that no column of S takes part in: the gates, the running maximum m,
// the normaliser n and the read-out's denominator.  One warp per (sequence, head) walks the tokens
// and leaves three numbers per token for the CTAs that own the columns; three more warps fetch the
// next tokens' q and k meanwhile and work out their gates' logarithms, which need no earlier token.
constexpr int NPL = (DIM + 31) / 32;          // entries of n per lane
constexpr int SCHUNK = DIM <= 64 ? 32 : DIM <= 128 ? 16 : DIM <= 256 ? 8 : DIM <= 512 ? 4 : 2;

template <typename T>
__global__ void __launch_bounds__(128) mlstm_scan_kernel(MlstmArgs a, IertBatchView b) {
  __shared__ __align__(16) float k_s[2][SCHUNK][DIM], q_s[2][SCHUNK][DIM], g_s[2][SCHUNK][2];
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, lane = threadIdx.x & 31;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const bool loader = threadIdx.x >= 32;
  const float qscale = 1.0f / sqrtf((float)DIM);
  const T* proj = (const T*)a.proj;
  auto fetch = [&](int buf, int tc, int tid, int nthreads) {
    const int n = min(SCHUNK, t1 - tc);
    if (sizeof(T) == 2 && DIM % 8 == 0 && a.ld % 8 == 0 && ((uintptr_t)a.proj & 15) == 0) {      // eight bf16 per load
      // every load of the chunk is issued before the first is converted and stored
      constexpr int ITER = (SCHUNK * (DIM / 8) * 2 + 96 - 1) / 96 > 0 ? (SCHUNK * (DIM / 8) * 2 + 96 - 1) / 96 : 1;     // key sizes below 8 never take this branch
      uint4 raw[ITER];
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 8) * 2) {
          const int which = x & 1, y = x >> 1;
          const int tt = y / (DIM / 8), d = 8 * (y - tt * (DIM / 8));
          raw[it] = *reinterpret_cast<const uint4*>(proj + (size_t)(tc + tt) * a.ld + (which ? a.H * DIM : 0) + head * DIM + d);
        }
      }
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 8) * 2) {
          const int which = x & 1, y = x >> 1;
          const int tt = y / (DIM / 8), d = 8 * (y - tt * (DIM / 8));
          const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[it]);
          float* dst = which ? &k_s[buf][tt][d] : &q_s[buf][tt][d];
          const float sc = which ? 1.f : qscale;
          const float2 f0 = __bfloat1622float2(p[0]), f1 = __bfloat1622float2(p[1]);
          const float2 f2 = __bfloat1622float2(p[2]), f3 = __bfloat1622float2(p[3]);
          *reinterpret_cast<float4*>(dst) = make_float4(f0.x * sc, f0.y * sc, f1.x * sc, f1.y * sc);
          *reinterpret_cast<float4*>(dst + 4) = make_float4(f2.x * sc, f2.y * sc, f3.x * sc, f3.y * sc);
        }
      }
    } else {
      for (int x = tid; x < n * DIM; x += nthreads) {
        const int tt = x / DIM, d = x - tt * DIM;
        const T* rowp = proj + (size_t)(tc + tt) * a.ld;
        q_s[buf][tt][d] = to_f32(rowp[head * DIM + d]) * qscale;
        k_s[buf][tt][d] = to_f32(rowp[a.H * DIM + head * DIM + d]);
      }
    }
    for (int tt = tid; tt < n; tt += nthreads) {
      const float zi = a.gates[(size_t)(tc + tt) * a.gld + head] + a.bi[head];
      const float zf = a.gates[(size_t)(tc + tt) * a.gld + a.H + head] + a.bf[head];
      g_s[buf][tt][0] = a.cap * tanhf(zi / a.cap);
      g_s[buf][tt][1] = logsigmoid_f(a.cap * tanhf(zf / a.cap));
    }
  };
  float* base = a.state + (size_t)slot * a.state_stride;
  float* ng = base + a.n_off + (size_t)head * DIM;
  float nn[NPL];
#pragma unroll
  for (int i = 0; i < NPL; ++i) nn[i] = lane + 32 * i < DIM ? ng[lane + 32 * i] : 0.f;
  float m = base[a.m_off + head];
  fetch(0, t0, threadIdx.x, blockDim.x);
  __syncthreads();
  int buf = 0;
  for (int tc = t0; tc < t1; tc += SCHUNK, buf ^= 1) {
    const int n = min(SCHUNK, t1 - tc);
    if (loader) {
      if (tc + SCHUNK < t1) fetch(buf ^ 1, tc + SCHUNK, threadIdx.x - 32, blockDim.x - 32);
    } else {
#pragma unroll 4
      for (int tt = 0; tt < SCHUNK; ++tt) {
        if (tt >= n) break;
        const float li = g_s[buf][tt][0], lf = g_s[buf][tt][1];
        const float m_new = fmaxf(lf + m, li);
        const float ea = expf(lf + m - m_new), eb = expf(li - m_new);
        m = m_new;
        float nq = 0.f;
#pragma unroll
        for (int i = 0; i < NPL; ++i) {
          const int d = lane + 32 * i;
          if (d < DIM) {
            nn[i] = fmaf(ea, nn[i], eb * k_s[buf][tt][d]);
            nq = fmaf(nn[i], q_s[buf][tt][d], nq);
          }
        }
        nq = warp_sum(nq);
        if (lane == 0) {
          float* c = a.coef + ((size_t)(tc + tt) * a.H + head) * 3;
          c[0] = ea; c[1] = eb; c[2] = fmaxf(fabsf(nq), expf(-m)) + 1e-6f;
        }
      }
    }
    __syncthreads();
  }
  if (!loader) {
#pragma unroll
    for (int i = 0; i < NPL; ++i) if (lane + 32 * i < DIM) ng[lane + 32 * i] = nn[i];
    if (lane == 0) base[a.m_off + head] = m;
  }
}

template <typename T, int R>
__global__ void __launch_bounds__(256 + LOADERS) mlstm_recur_kernel(MlstmArgs a, IertBatchView b) {
  constexpr int RPT = (DIM + R - 1) / R;
  __shared__ __align__(16) float k_s[2][CHUNK][DIM], q_s[2][CHUNK][DIM], v_s[2][CHUNK][256], c_s[2][CHUNK][3];
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * a.cols;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const int workers = blockDim.x - LOADERS;
  const bool loader = (int)threadIdx.x >= workers;
  const int col = threadIdx.x / R, r = threadIdx.x % R;
  const int j = c0 + col;
  const bool live = !loader && col < a.cols && j < a.V;
  const float qscale = 1.0f / sqrtf((float)DIM);
  const T* proj = (const T*)a.proj;
  auto fetch = [&](int buf, int tc, int tid, int nthreads) {
    const int n = min(CHUNK, t1 - tc);
    if (sizeof(T) == 2 && DIM % 8 == 0 && a.ld % 8 == 0 && ((uintptr_t)a.proj & 15) == 0) {      // eight bf16 per load
      // every load of the chunk is issued before the first is converted and stored
      constexpr int ITER = (CHUNK * (DIM / 8) * 2 + LOADERS - 1) / LOADERS > 0 ? (CHUNK * (DIM / 8) * 2 + LOADERS - 1) / LOADERS : 1;
      uint4 raw[ITER];
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 8) * 2) {
          const int which = x & 1, y = x >> 1;
          const int tt = y / (DIM / 8), d = 8 * (y - tt * (DIM / 8));
          raw[it] = *reinterpret_cast<const uint4*>(proj + (size_t)(tc + tt) * a.ld + (which ? a.H * DIM : 0) + head * DIM + d);
        }
      }
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 8) * 2) {
          const int which = x & 1, y = x >> 1;
          const int tt = y / (DIM / 8), d = 8 * (y - tt * (DIM / 8));
          const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[it]);
          float* dst = which ? &k_s[buf][tt][d] : &q_s[buf][tt][d];
          const float sc = which ? 1.f : qscale;
          const float2 f0 = __bfloat1622float2(p[0]), f1 = __bfloat1622float2(p[1]);
          const float2 f2 = __bfloat1622float2(p[2]), f3 = __bfloat1622float2(p[3]);
          *reinterpret_cast<float4*>(dst) = make_float4(f0.x * sc, f0.y * sc, f1.x * sc, f1.y * sc);
          *reinterpret_cast<float4*>(dst + 4) = make_float4(f2.x * sc, f2.y * sc, f3.x * sc, f3.y * sc);
        }
      }
    } else {
      for (int x = tid; x < n * DIM; x += nthreads) {
        const int tt = x / DIM, d = x - tt * DIM;
        const T* rowp = proj + (size_t)(tc + tt) * a.ld;
        q_s[buf][tt][d] = to_f32(rowp[head * DIM + d]) * qscale;
        k_s[buf][tt][d] = to_f32(rowp[a.H * DIM + head * DIM + d]);
      }
    }
    for (int x = tid; x < n * a.cols; x += nthreads) {
      const int tt = x / a.cols, cc = x - tt * a.cols;
      v_s[buf][tt][cc] = c0 + cc < a.V ? to_f32(proj[(size_t)(tc + tt) * a.ld + 2 * a.H * DIM + head * a.V + c0 + cc]) : 0.f;
    }
    if (tid < n * 3) c_s[buf][tid / 3][tid % 3] = a.coef[((size_t)(tc + tid / 3) * a.H + head) * 3 + tid % 3];
  };
  float* Sg = a.state + (size_t)slot * a.state_stride + a.s_off + (size_t)head * DIM * a.V;
  float S[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int d = i * R + r;
    S[i] = (live && d < DIM) ? Sg[(size_t)d * a.V + j] : 0.f;
  }
  fetch(0, t0, threadIdx.x, blockDim.x);
  __syncthreads();
  int buf = 0;
  for (int tc = t0; tc < t1; tc += CHUNK, buf ^= 1) {
    const int n = min(CHUNK, t1 - tc);
    if (loader) {
      if (tc + CHUNK < t1) fetch(buf ^ 1, tc + CHUNK, threadIdx.x - workers, LOADERS);
    } else {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) {
        if (tt >= n) break;
        const float ea = c_s[buf][tt][0], eb = c_s[buf][tt][1], den = c_s[buf][tt][2];
        const float bv = eb * (live ? v_s[buf][tt][col] : 0.f);
        float oq = 0.f;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int d = i * R + r;
          const float kd = d < DIM ? k_s[buf][tt][d] : 0.f, qd = d < DIM ? q_s[buf][tt][d] : 0.f;
          S[i] = fmaf(ea, S[i], kd * bv);
          oq = fmaf(S[i], qd, oq);
        }
        oq = group_sum<R>(oq);
        if (live && r == 0) a.o[(size_t)(tc + tt) * a.H * a.V + (size_t)head * a.V + j] = oq / den;
      }
    }
    __syncthreads();
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int d = i * R + r;
      if (d < DIM) Sg[(size_t)d * a.V + j] = S[i];
    }
  }
}

struct WkvArgs {
  const float* x;        // [T, ld] fp32: r [H*DIM] | k [H*DIM] | v [H*V] | ... (the projections)
  long long ld;
  const float* decay;    // [T, H*DIM] fp32: w, the factor of each row of S
  const float* u;        // [H, DIM] fp32: the current token's bonus
  float* state;          // per slot at s_off: S [H, DIM, V]
  long long state_stride, s_off;
  float* o;              // [T, H*V] fp32
  int H, V, cols;
};

template <int R>
__global__ void __launch_bounds__(256 + LOADERS) wkv_recur_kernel(WkvArgs a, IertBatchView b) {
  constexpr int RPT = (DIM + R - 1) / R;
  __shared__ __align__(16) float r_s[2][CHUNK][DIM], k_s[2][CHUNK][DIM], w_s[2][CHUNK][DIM], v_s[2][CHUNK][256];
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * a.cols;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const int workers = blockDim.x - LOADERS;
  const bool loader = (int)threadIdx.x >= workers;
  const int col = threadIdx.x / R, r = threadIdx.x % R;
  const int j = c0 + col;
  const bool live = !loader && col < a.cols && j < a.V;
  const int HD = a.H * DIM;
  auto fetch = [&](int buf, int tc, int tid, int nthreads) {
    const int n = min(CHUNK, t1 - tc);
    if (DIM % 4 == 0 && a.ld % 4 == 0 && ((uintptr_t)a.x & 15) == 0 && ((uintptr_t)a.decay & 15) == 0) {     // 16-byte loads
      // every load of the chunk is issued before the first is stored (a loader's loads are all it waits for)
      constexpr int ITER = (CHUNK * (DIM / 4) + LOADERS - 1) / LOADERS > 0 ? (CHUNK * (DIM / 4) + LOADERS - 1) / LOADERS : 1;
      float4 rv[ITER], kv[ITER], wv[ITER];
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 4)) {
          const int tt = x / (DIM / 4), d = 4 * (x - tt * (DIM / 4));
          const float* rowp = a.x + (size_t)(tc + tt) * a.ld + head * DIM + d;
          rv[it] = *reinterpret_cast<const float4*>(rowp);
          kv[it] = *reinterpret_cast<const float4*>(rowp + HD);
          wv[it] = *reinterpret_cast<const float4*>(a.decay + (size_t)(tc + tt) * HD + head * DIM + d);
        }
      }
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const int x = tid + it * nthreads;
        if (x < n * (DIM / 4)) {
          const int tt = x / (DIM / 4), d = 4 * (x - tt * (DIM / 4));
          *reinterpret_cast<float4*>(&r_s[buf][tt][d]) = rv[it];
          *reinterpret_cast<float4*>(&k_s[buf][tt][d]) = kv[it];
          *reinterpret_cast<float4*>(&w_s[buf][tt][d]) = wv[it];
        }
      }
    } else {
      for (int x = tid; x < n * DIM; x += nthreads) {
        const int tt = x / DIM, d = x - tt * DIM;
        const float* rowp = a.x + (size_t)(tc + tt) * a.ld + head * DIM + d;
        r_s[buf][tt][d] = rowp[0];
        k_s[buf][tt][d] = rowp[HD];
        w_s[buf][tt][d] = a.decay[(size_t)(tc + tt) * HD + head * DIM + d];
      }
    }
    for (int x = tid; x < n * a.cols; x += nthreads) {
      const int tt = x / a.cols, cc = x - tt * a.cols;
      v_s[buf][tt][cc] = c0 + cc < a.V ? a.x[(size_t)(tc + tt) * a.ld + 2 * HD + head * a.V + c0 + cc] : 0.f;
    }
  };
  float* Sg = a.state + (size_t)slot * a.state_stride + a.s_off + (size_t)head * DIM * a.V;
  float S[RPT], u[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int d = i * R + r;
    S[i] = (live && d < DIM) ? Sg[(size_t)d * a.V + j] : 0.f;
    u[i] = d < DIM ? a.u[head * DIM + d] : 0.f;
  }
  fetch(0, t0, threadIdx.x, blockDim.x);
  __syncthreads();
  int buf = 0;
  for (int tc = t0; tc < t1; tc += CHUNK, buf ^= 1) {
    const int n = min(CHUNK, t1 - tc);
    if (loader) {
      if (tc + CHUNK < t1) fetch(buf ^ 1, tc + CHUNK, threadIdx.x - workers, LOADERS);
    } else {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) {
        if (tt >= n) break;
        const float vj = live ? v_s[buf][tt][col] : 0.f;
        float oq = 0.f;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int d = i * R + r;
          const float kd = d < DIM ? k_s[buf][tt][d] : 0.f, rd = d < DIM ? r_s[buf][tt][d] : 0.f;
          const float wd = d < DIM ? w_s[buf][tt][d] : 0.f;
          const float kv = kd * vj;
          oq = fmaf(rd, fmaf(u[i], kv, S[i]), oq);
          S[i] = fmaf(wd, S[i], kv);
        }
        oq = group_sum<R>(oq);
        if (live && r == 0) a.o[(size_t)(tc + tt) * a.H * a.V + (size_t)head * a.V + j] = oq;
      }
    }
    __syncthreads();
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int d = i * R + r;
      if (d < DIM) Sg[(size_t)d * a.V + j] = S[i];
    }
  }
}

#if DIM == 64               // (at 128 the ring would not fit beside the scaled rows in the shared memory that needs no opt-in)
// Prompts, eight tokens at a time, as for the delta rule above.  With W_i = w_1 .. w_i (per row of S) the state in front of the
// chunk S gives
//   o_i = (W_(i-1) r_i).S + sum_{j < i} (sum_d r_i k_j w_(j+1) .. w_(i-1)) v_j + (r_i.(u k_i)) v_i
//   S  <- W_8 S + sum_j (w_(j+1) .. w_8 k_j) v_j^T
// There is no chain inside a chunk at all.  The products of two tokens (decays multiplied, never divided) come from a kernel in
// front with a block per chunk and head; here a loader thread per row of S brings the rows through a ring and scales them.
constexpr int WLOAD = DIM;

// pairs[token][head][8]: row i of the chunk's products with the tokens j <= i.  Thread d: row d's share, then summed over the rows.
__global__ void __launch_bounds__(DIM) wkv_pairs_kernel(WkvArgs a, float* __restrict__ pairs, IertBatchView b) {
  __shared__ float sum_s[DIM / 32][36];
  pdl_wait();                                                    // (no early start for the kernel behind, as above)
  int tc, t1;
  if (!chunk_of(b, blockIdx.x, tc, t1)) return;
  const int head = blockIdx.y, d = threadIdx.x, lane = d & 31, HD = a.H * DIM, n = min(CT, t1 - tc);
  const float bonus = a.u[head * DIM + d];
  float r[CT], k[CT], w[CT];
#pragma unroll
  for (int t = 0; t < CT; ++t) {
    const size_t tok = tc + min(t, n - 1);
    const float* row = a.x + tok * a.ld + head * DIM + d;
    r[t] = row[0];
    k[t] = row[HD];
    w[t] = a.decay[tok * HD + head * DIM + d];
  }
  float p[36];                                                   // pair (i, j <= i) at i (i + 1) / 2 + j
#pragma unroll
  for (int j = 0; j < CT; ++j) {
    p[j * (j + 1) / 2 + j] = r[j] * (bonus * k[j]);
    float e = k[j];
#pragma unroll
    for (int i = j + 1; i < CT; ++i) {
      p[i * (i + 1) / 2 + j] = r[i] * e;
      e *= w[i];
    }
  }
  // over the warp's rows: 32 of the sums spread over the lanes, the other four by full butterflies
#pragma unroll
  for (int half = 16; half > 0; half >>= 1) {
    const bool upper = lane & half;
#pragma unroll
    for (int m = 0; m < half; ++m) {
      const float send = upper ? p[m] : p[m + half], keep = upper ? p[m + half] : p[m];
      p[m] = keep + __shfl_xor_sync(0xffffffffu, send, half);
    }
  }
#pragma unroll
  for (int m = 32; m < 36; ++m) p[m] = warp_sum(p[m]);
  sum_s[d / 32][lane] = p[0];
  if (lane < 4) sum_s[d / 32][32 + lane] = lane == 0 ? p[32] : lane == 1 ? p[33] : lane == 2 ? p[34] : p[35];
  __syncthreads();
  const int i = d / CT, j = d % CT;                              // (64 threads: one per entry)
  if (i < n) {
    float t = 0.f;
    if (j <= i) {
      t = sum_s[0][i * (i + 1) / 2 + j];
#pragma unroll
      for (int x = 1; x < DIM / 32; ++x) t += sum_s[x][i * (i + 1) / 2 + j];
    }
    pairs[((size_t)(tc + i) * a.H + head) * CT + j] = t;
  }
}

__global__ void __launch_bounds__(CWORK + WLOAD) wkv_chunk_kernel(WkvArgs a, const float* __restrict__ pairs, IertBatchView b) {
  __shared__ __align__(16) float raw_s[RING][3][CT][DIM];        // r, k, w as they are in memory
  __shared__ __align__(16) float v_s[RING][CT][CCOLS], p_s[RING][CT][CT], rt_s[2][CT][DIM], kt_s[2][CT][DIM], wc_s[2][DIM];
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * CCOLS;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const int n_chunks = (t1 - t0 + CT - 1) / CT, HD = a.H * DIM;

  if (threadIdx.x >= CWORK) {
    // ---------------- loaders: three chunks ahead; thread d scales row d ----------------
    const int d = threadIdx.x - CWORK;
    auto ask = [&](int n) {
      if (n < n_chunks) {
        const int tc = t0 + n * CT, buf = n % RING;
        for (int x = d; x < 3 * CT * DIM / 4; x += WLOAD) {
          const int which = x / (CT * DIM / 4), t = x / (DIM / 4) % CT, e = 4 * (x % (DIM / 4));
          const bool in = tc + t < t1;
          const size_t tok = in ? tc + t : t0;
          copy16(&raw_s[buf][which][t][e], which < 2 ? a.x + tok * a.ld + which * HD + head * DIM + e : a.decay + tok * HD + head * DIM + e, in);
        }
        for (int x = d; x < CT * (CCOLS + CT) / 4; x += WLOAD) {
          const bool of_v = x < CT * CCOLS / 4;
          const int y = of_v ? x : x - CT * CCOLS / 4;
          const int t = of_v ? y / (CCOLS / 4) : y / (CT / 4), e = 4 * (of_v ? y % (CCOLS / 4) : y % (CT / 4));
          const bool in = tc + t < t1, col = c0 + e < a.V;
          const size_t tok = in ? tc + t : t0;
          if (of_v) copy16(&v_s[buf][t][e], a.x + tok * a.ld + 2 * HD + (col ? head * a.V + c0 + e : 0), in && col);
          else copy16(&p_s[buf][t][e], pairs + (tok * a.H + head) * CT + e, in);
        }
      }
      copies_commit();
    };
    auto scale = [&](int n) {                                    // a token beyond the sequence: zeros, decay 1
      const int buf = n % RING, out = n & 1, left = t1 - (t0 + n * CT);
      float w[CT], pw = 1.f, sw = 1.f;
#pragma unroll
      for (int t = 0; t < CT; ++t) w[t] = t < left ? raw_s[buf][2][t][d] : 1.f;
#pragma unroll
      for (int t = 0; t < CT; ++t) { rt_s[out][t][d] = raw_s[buf][0][t][d] * pw; pw *= w[t]; }
      wc_s[out][d] = pw;
#pragma unroll
      for (int t = CT - 1; t >= 0; --t) { kt_s[out][t][d] = raw_s[buf][1][t][d] * sw; sw *= w[t]; }
    };
    for (int n = 0; n < RING - 1; ++n) ask(n);
    copies_wait<RING - 2>();
    asm volatile("bar.sync 1, %0;" ::"n"(WLOAD) : "memory");     // every loader's copies of chunk 0
    scale(0);
    __syncthreads();
    for (int n = 0; n < n_chunks; ++n) {
      copies_wait<RING - 3>();                                   // chunk n + 1 has arrived ...
      asm volatile("bar.sync 1, %0;" ::"n"(WLOAD) : "memory");   // ... for all loaders
      if (n + 1 < n_chunks) scale(n + 1);
      ask(n + RING - 1);                 // its place: read by the workers before the last barrier, scaled from two chunks ago
      __syncthreads();
    }
    return;
  }

  // ---------------- workers ----------------
  const int r = threadIdx.x % CL, grp = threadIdx.x / CL, j0 = c0 + grp * CG;
  const bool live = j0 < a.V;
  const int i_own = r >> 1, col2 = 2 * (r & 1);      // the token and the two columns whose read-out this lane ends with
  float* Sg = a.state + (size_t)slot * a.state_stride + a.s_off + (size_t)head * DIM * a.V + j0;
  float2 S[CP][CG];
  load_rows(S, Sg, a.V, r, live);
  __syncthreads();
  for (int n = 0; n < n_chunks; ++n) {
    const int buf = n & 1, ring = n % RING;
    float v[16][CG];                                  // [8] used
#pragma unroll
    for (int t = 0; t < CT; ++t) {
      float2 rr[CP];
      own_rows(rr, rt_s[buf][t], r);
#pragma unroll
      for (int c = 0; c < CG; ++c) {
        float2 o = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < CP; ++i) o = fma2(S[i][c], rr[i], o);
        v[t][c] = o.x + o.y;
      }
    }
    halve<4, 8>(v, r & 8);
    halve<2, 4>(v, r & 4);
    halve<1, 2>(v, r & 2);
    const bool odd = r & 1;
    float o[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float send = odd ? v[0][c] : v[0][c + 2], keep = odd ? v[0][c + 2] : v[0][c];
      o[c] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
    }
    float pr[CT];
    *reinterpret_cast<float4*>(pr) = *reinterpret_cast<const float4*>(&p_s[ring][i_own][0]);
    *reinterpret_cast<float4*>(pr + 4) = *reinterpret_cast<const float4*>(&p_s[ring][i_own][4]);
    float2 wc[CP];
    own_rows(wc, wc_s[buf], r);
#pragma unroll
    for (int i = 0; i < CP; ++i)
#pragma unroll
      for (int c = 0; c < CG; ++c) S[i][c] = mul2(S[i][c], wc[i]);
#pragma unroll
    for (int j = 0; j < CT; ++j) {
      const float4 f = *reinterpret_cast<const float4*>(&v_s[ring][j][grp * CG]);
      if (j <= i_own) {
        o[0] = fmaf(pr[j], odd ? f.z : f.x, o[0]);
        o[1] = fmaf(pr[j], odd ? f.w : f.y, o[1]);
      }
      const float vv[CG] = {f.x, f.y, f.z, f.w};
      float2 kt[CP];
      own_rows(kt, kt_s[buf][j], r);
#pragma unroll
      for (int c = 0; c < CG; ++c) {
        const float2 v2 = make_float2(vv[c], vv[c]);
#pragma unroll
        for (int i = 0; i < CP; ++i) S[i][c] = fma2(kt[i], v2, S[i][c]);
      }
    }
    if (live && t0 + n * CT + i_own < t1)
      *reinterpret_cast<float2*>(a.o + (size_t)(t0 + n * CT + i_own) * a.H * a.V + (size_t)head * a.V + j0 + col2) = make_float2(o[0], o[1]);
    __syncthreads();
  }
  if (live) store_rows(S, Sg, a.V, r);
}
#endif

// Lanes per column: the fewest that give the device about eight warps per SM (at most 32), and columns per
// CTA so that a CTA has up to 256 computing threads.  (Measured at 32 heads of 128 x 128, one prompt of 2,048
// tokens: 8 lanes per column 1.08 ms, 16 lanes 0.91 ms, 32 lanes 1.42 ms per layer.)
#if IERT_CHUNKED
// Prompts go eight tokens at a time; steps of few tokens per sequence token after token: a chunk costs what eight tokens cost, the kernel
// in front is one launch more, and such a step is bound by reading and writing the state.  Where the line lies (layers at 4,096, sequences of
// equal length, chunks / token after token, us):
//   delta rule, 16 tokens a sequence: one sequence 56 / 54, eight 133 / 132, 32 314 / 313, 128 930 / 961; four tokens 51 / 46, 93 / 85,
//   201 / 173, 577 / 493; twelve 55 / 52, 124 / 117, 280 / 255, 882 / 817; 64 87 / 93, 254 / 282, 693 / 763;
//   decays per channel: one sequence of 4 to 32 tokens 71 / 70 to 109 / 110, two of 8 82 / 81, four of 8 110 / 113, eight of 4 114 / 118 and of
//   16 138 / 165, 32 of 4 170 / 185.
bool chunked(const IertBatchView* b, int tokens_a_sequence, int tokens) {
  const char* off = getenv("IERT_RECURRENT_LANES");                  // (a forced number of lanes asks for the other kernels)
  return !(off && atoi(off) >= 1) && b->n_tokens >= tokens && b->n_tokens >= (long long)tokens_a_sequence * b->n_seqs;
}
#endif

struct Split { int lanes, cols; };
Split pick_split(int n_seqs, int H, int V) {
  const long long want = 8LL * 32 * iert_sm_count_cached();          // threads
  int lanes = R_MIN;
  while (lanes < 32 && (long long)n_seqs * H * V * lanes < want) lanes *= 2;
  if (const char* forced = getenv("IERT_RECURRENT_LANES")) {         // for tests and measurements: 1, 2, ... 32
    const int f = atoi(forced);
    if (f >= 1) { lanes = R_MIN; while (lanes < 32 && lanes < f) lanes *= 2; }
  }
  int cols = 256 / lanes;
  if (cols > V) cols = V;
  return {lanes, cols};
}

}  // namespace

IERT_API int iert_recurrent_dim() { return DIM; }

#define IERT_BY_LANES(L, CALL)                                       \
  switch (L) {                                                       \
    case 1: { constexpr int RR = 1 < R_MIN ? R_MIN : 1; CALL; } break;    \
    case 2: { constexpr int RR = 2 < R_MIN ? R_MIN : 2; CALL; } break;    \
    case 4: { constexpr int RR = 4 < R_MIN ? R_MIN : 4; CALL; } break;    \
    case 8: { constexpr int RR = 8 < R_MIN ? R_MIN : 8; CALL; } break;    \
    case 16: { constexpr int RR = 16 < R_MIN ? R_MIN : 16; CALL; } break; \
    default: { constexpr int RR = 32; CALL; } break;                 \
  }

// Scratch (floats) of the recurrences over n_tokens tokens and H heads: the products of tokens with one another.
IERT_API long long iert_recurrent_scratch_floats(int n_tokens, int H) { return (long long)n_tokens * H * 20; }

// scratch: as many floats as above, or null (then tokens go one after another)
IERT_API int iert_delta_recur(const float* qkv, const float* beta, const float* decay, float* state,
                              long long state_stride, long long s_off, float* o, float* scratch, int G, int H, int V,
                              const IertBatchView* batch, cudaStream_t stream) {
  if (batch->n_seqs <= 0 || batch->n_tokens <= 0) return IERT_OK;
  if (G <= 0 || H <= 0 || H % G || V <= 0 || H > 65535) return IERT_BAD_ARGUMENT;
#if IERT_CHUNKED
  if (scratch && chunked(batch, 16, 16) && V % 4 == 0 && (2 * G * DIM + H * V) % 4 == 0 && state_stride % 4 == 0 && s_off % 4 == 0 &&
      (((uintptr_t)qkv | (uintptr_t)state | (uintptr_t)o | (uintptr_t)scratch) & 15) == 0) {
    DeltaArgs a = {qkv, beta, decay, state, state_stride, s_off, o, G, H, V, CCOLS};
    launch_dep(delta_coef_kernel, dim3(batch->n_tokens / CT + batch->n_seqs, G), dim3(128), 0, stream, a, scratch, *batch);
    launch_dep(delta_chunk_kernel, dim3(batch->n_seqs, H, (V + CCOLS - 1) / CCOLS), dim3(CWORK + 32), 0, stream, a, (const float*)scratch, *batch);
    return iert_check_launch("delta_recur");
  }
#endif
  const Split sp = pick_split(batch->n_seqs, H, V);
  DeltaArgs a = {qkv, beta, decay, state, state_stride, s_off, o, G, H, V, sp.cols};
  dim3 grid(batch->n_seqs, H, (V + sp.cols - 1) / sp.cols);
  const int threads = ((sp.cols * sp.lanes + 31) / 32) * 32 + LOADERS;
  IERT_BY_LANES(sp.lanes, launch_dep(delta_recur_kernel<RR>, grid, dim3(threads), 0, stream, a, *batch));
  return iert_check_launch("delta_recur");
}

// x: fp32 [T, ld] = r [H*DIM] | k [H*DIM] | v [H*V] | ...; decay fp32 [T, H*DIM]; u fp32 [H, DIM]; o fp32 [T, H*V].
IERT_API int iert_wkv_recur(const float* x, long long ld, const float* decay, const float* u, float* state,
                            long long state_stride, long long s_off, float* o, float* scratch, int H, int V, const IertBatchView* batch,
                            cudaStream_t stream) {
  if (batch->n_seqs <= 0 || batch->n_tokens <= 0) return IERT_OK;
  if (H <= 0 || V <= 0 || H > 65535 || ld < (long long)2 * H * DIM + (long long)H * V) return IERT_BAD_ARGUMENT;
#if DIM == 64
  if (scratch && chunked(batch, 4, 32) && V % 4 == 0 && ld % 4 == 0 && state_stride % 4 == 0 && s_off % 4 == 0 &&
      (((uintptr_t)x | (uintptr_t)decay | (uintptr_t)state | (uintptr_t)o | (uintptr_t)scratch) & 15) == 0) {
    WkvArgs a = {x, ld, decay, u, state, state_stride, s_off, o, H, V, CCOLS};
    launch_dep(wkv_pairs_kernel, dim3(batch->n_tokens / CT + batch->n_seqs, H), dim3(DIM), 0, stream, a, scratch, *batch);
    launch_dep(wkv_chunk_kernel, dim3(batch->n_seqs, H, (V + CCOLS - 1) / CCOLS), dim3(CWORK + WLOAD), 0, stream, a, (const float*)scratch, *batch);
    return iert_check_launch("wkv_recur");
  }
#endif
  const Split sp = pick_split(batch->n_seqs, H, V);
  WkvArgs a = {x, ld, decay, u, state, state_stride, s_off, o, H, V, sp.cols};
  dim3 grid(batch->n_seqs, H, (V + sp.cols - 1) / sp.cols);
  const int threads = ((sp.cols * sp.lanes + 31) / 32) * 32 + LOADERS;
  IERT_BY_LANES(sp.lanes, launch_dep(wkv_recur_kernel<RR>, grid, dim3(threads), 0, stream, a, *batch));
  return iert_check_launch("wkv_recur");
}

IERT_API int iert_mlstm_recur(const void* proj, int dtype, long long ld, const float* gates, long long gld,
                              const float* bi, const float* bf, float cap, float* state, long long state_stride,
                              long long s_off, long long n_off, long long m_off, float* coef, float* o, int H, int V,
                              const IertBatchView* batch, cudaStream_t stream) {
  if (batch->n_seqs <= 0 || batch->n_tokens <= 0) return IERT_OK;
  if (H <= 0 || V <= 0 || H > 65535 || !(cap > 0.f) || (dtype != IERT_F32 && dtype != IERT_BF16)) return IERT_BAD_ARGUMENT;
  const Split sp = pick_split(batch->n_seqs, H, V);
  MlstmArgs a = {proj, ld, gates, gld, bi, bf, cap, state, state_stride, s_off, n_off, m_off, coef, o, H, V, sp.cols};
  dim3 grid(batch->n_seqs, H, (V + sp.cols - 1) / sp.cols);
  const int threads = ((sp.cols * sp.lanes + 31) / 32) * 32 + LOADERS;
  if (dtype == IERT_F32) {
    launch_dep(mlstm_scan_kernel<float>, dim3(batch->n_seqs, H), dim3(128), 0, stream, a, *batch);
    IERT_BY_LANES(sp.lanes, (launch_dep(mlstm_recur_kernel<float, RR>, grid, dim3(threads), 0, stream, a, *batch)));
  } else {
    launch_dep(mlstm_scan_kernel<__nv_bfloat16>, dim3(batch->n_seqs, H), dim3(128), 0, stream, a, *batch);
    IERT_BY_LANES(sp.lanes, (launch_dep(mlstm_recur_kernel<__nv_bfloat16, RR>, grid, dim3(threads), 0, stream, a, *batch)));
  }
  return iert_check_launch("mlstm_recur");
}
