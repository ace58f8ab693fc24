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

// ---- prompts: sixteen tokens at a time, on the tensor cores ------------------------------------------------------------
// Token after token, a step's time is the latency of its chain (dot product, shuffles, update: about 680 cycles a token), not its
// work.  Over a chunk of 16 tokens with decays g and G_i = g_1 .. g_i, the state in front of the chunk S and u_i as above:
//
//   S_i = G_i S + sum_{j <= i} (G_i / G_j) k_j u_j      so      u_i + sum_{j < i} A_ij u_j = x_i = beta_i (v_i - G_i k_i.S),
//   A_ij = beta_i (G_i / G_j) (k_i.k_j)                          u = T x,  T = (1 + A)^-1  (lower triangular)
//   o_i = G_i q_i.S + sum_{j <= i} P_ij u_j,  P_ij = (G_i / G_j) (q_i.k_j)
//
// T and P (the same for all columns; ratios are products of the decays between, never quotients) come from a kernel in front with a
// block per chunk and key head.  What is left is products of matrices: k.S, q.S, T x, P u and the update k^T u, on mma.sync m16n8k16.
// The state is kept transposed, S^T [16 columns x rows], in the accumulator layout of one warp: as the left operand of k.S and
// q.S it needs no exchange between lanes, and x and u come out as left operands of the next product.
//
// Everything stays fp32: an operand is the sum of three bf16 numbers (the nearest, the nearest to the remainder, the rest), a
// product is the six partial products of weight 2^-16 and more, the largest in an accumulator of its own and no accumulator over
// more than DIM / 2 numbers; these sums are added to fp32 registers by rounded additions (the three products left out come to 2^-24).
// mma.sync runs at 1,020 multiply-adds per clock and SM here, so six products are worth 170 against 124 for FFMA, and there are
// no dot products to add over lanes (15 shuffles per sum of 16 lanes before).
//
// A block owns 32 columns: four warps compute, each 16 columns x half of the rows (the halves of k.S and q.S are exchanged through
// shared memory), four bring q, k, v and the coefficients and split them.  2,048 tokens, 32 heads of 128 x 128 (128 blocks): 200 to
// 212 us; eight tokens at a time with FFMA, a thread holding 8 rows of four columns, took 344.  What bounds it is the chain
// k.S - x - u - S of a warp, about 2,500 cycles a chunk, in half of which the tensor pipe is active (162 mma.sync of 8 cycles): nothing else of
// that warp's scheduler has as much to do.  Other splits were no faster: q.S and P u in warps of their own with the state's parts
// through shared memory 222, quarters of the rows in twice the warps 261 (236 with the column groups half a chunk apart).
#define IERT_CHUNKED (DIM == 64 || DIM == 128)                // (larger sizes would not fit the registers)
#if IERT_CHUNKED
constexpr int CT = 16, CCOLS = 32, RING = 4;                  // tokens of a chunk, columns of a block, chunks in shared memory
constexpr int CLOAD = 128;                                    // loading threads
constexpr int OPROW = DIM + 8;                                // numbers from row to row of an operand tile: 8 rows meet no bank twice
constexpr int VROW = CCOLS + 4;
// per token and head: 16 of T, 16 of P, then beta_i, G_i, G_16 / G_i, and G_16 at the chunk's first token
constexpr int COEF = 36, CROW = 40;
constexpr int TPROW = 24;                                     // rows of 16 coefficients as operands

template <bool FIRST>      // d = a b (+ d)
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (FIRST)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (Volatile, so that they stay behind the barriers in front of them; the tiles are other threads' writes, so this thread's own accesses may move past.)
template <bool TRANS>
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// Two numbers as pairs of bf16 numbers p[0] + p[1] + p[2]; every remainder is exact, but for bits below 2^-133, bf16's smallest number, which are
// lost (an error of 2^-134 at most; fp32 keeps bits down to 2^-149).  The first two parts stop at bf16's largest finite number: what rounds beyond
// it (3.39e38 and more) would leave a remainder of the other sign without end.  So an infinity is (largest, largest, infinity), whose products are
// the infinities that they are in fp32, and a NaN stays one.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 d;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ void split2(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  auto nearest = [](float2 f) {
    const __nv_bfloat162 two = __floats2bfloat162_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&two);
  };
  auto nearest_finite = [](float2 f) {
    uint32_t two;
    asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(two) : "f"(f.y), "f"(f.x));
    return two;
  };
  auto wide = [](uint32_t p) { return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u)); };
  float2 f = make_float2(x, y);
  p0 = nearest_finite(f);
  f = sub2(f, wide(p0));
  p1 = nearest_finite(f);
  p2 = nearest(sub2(f, wide(p1)));
}
// Two neighbouring accumulator tiles [16 x 8] as the three parts of a left operand [16 x 16].
struct Left { uint32_t p[3][4]; };
__device__ __forceinline__ void left_of(Left& a, const float (&t0)[4], const float (&t1)[4]) {
  split2(t0[0], t0[1], a.p[0][0], a.p[1][0], a.p[2][0]);
  split2(t0[2], t0[3], a.p[0][1], a.p[1][1], a.p[2][1]);
  split2(t1[0], t1[1], a.p[0][2], a.p[1][2], a.p[2][2]);
  split2(t1[2], t1[3], a.p[0][3], a.p[1][3], a.p[2][3]);
}
// A product's sums: the main one (first parts), first with second parts, and the rest.  (Sums of their own so that a product does not wait for the
// one in front of it: an mma.sync is issued every 8 clocks and takes 21.)
struct Sums {
  float m[4], a[4], b[4];
  __device__ __forceinline__ float2 two(int i) const {
    return add2(make_float2(m[2 * i], m[2 * i + 1]), add2(make_float2(a[2 * i], a[2 * i + 1]), make_float2(b[2 * i], b[2 * i + 1])));
  }
  __device__ __forceinline__ void all(float (&o)[4]) const {
    const float2 x = two(0), y = two(1);
    o[0] = x.x; o[1] = x.y; o[2] = y.x; o[3] = y.y;
  }
};
// The six products of a left operand with two right operands (tiles of 8 outputs), r[part][4] as ldmatrix brings them.
template <bool FIRST>
__device__ __forceinline__ void six_by_two(Sums& s0, Sums& s1, const Left& l, const uint32_t (&r)[3][4]) {
  mma16816<FIRST>(s0.b, l.p[0], r[2][0], r[2][1]); mma16816<FIRST>(s1.b, l.p[0], r[2][2], r[2][3]);
  mma16816<FIRST>(s0.a, l.p[0], r[1][0], r[1][1]); mma16816<FIRST>(s1.a, l.p[0], r[1][2], r[1][3]);
  mma16816<false>(s0.b, l.p[2], r[0][0], r[0][1]); mma16816<false>(s1.b, l.p[2], r[0][2], r[0][3]);
  mma16816<FIRST>(s0.m, l.p[0], r[0][0], r[0][1]); mma16816<FIRST>(s1.m, l.p[0], r[0][2], r[0][3]);
  mma16816<false>(s0.b, l.p[1], r[1][0], r[1][1]); mma16816<false>(s1.b, l.p[1], r[1][2], r[1][3]);
  mma16816<false>(s0.a, l.p[1], r[0][0], r[0][1]); mma16816<false>(s1.a, l.p[1], r[0][2], r[0][3]);
}
// Three parts of an operand tile whose rows are tokens, as two right operands.  TRANS: the tokens are summed over (k^T u); else they are
// the outputs (k.S).  `tile`: part 0, first row, first column.
template <bool TRANS>
__device__ __forceinline__ void right_of(uint32_t (&r)[3][4], const __nv_bfloat16* tile, int ld, int lane) {
  const int row = TRANS ? (lane & 7) + (((lane >> 3) & 1) << 3) : (lane & 7) + ((lane >> 4) << 3);
  const int col = TRANS ? (lane >> 4) * 8 : ((lane >> 3) & 1) * 8;
#pragma unroll
  for (int p = 0; p < 3; ++p) ldsm4<TRANS>(r[p], tile + (p * CT + row) * ld + col);
}
// Rows of coefficients of eight tokens (`tile`: part 0, first row) as a right operand, and the sums over the chunk's tokens of coefficient times x.
struct Rows { uint32_t p[3][2]; };
__device__ __forceinline__ void rows_of(Rows& b, const __nv_bfloat16* tile, int lane) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(tile + (p * CT + (lane & 7)) * TPROW + ((lane >> 3) & 1) * 8);
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(b.p[p][0]), "=r"(b.p[p][1]) : "r"(at));
  }
}
__device__ __forceinline__ void six_of_rows(float (&o)[4], const Left& l, const Rows& b) {
  float m[4], s0[4], s1[4];
  mma16816<true>(m, l.p[0], b.p[0][0], b.p[0][1]);
  mma16816<true>(s0, l.p[0], b.p[2][0], b.p[2][1]);
  mma16816<true>(s1, l.p[0], b.p[1][0], b.p[1][1]);
  mma16816<false>(s0, l.p[2], b.p[0][0], b.p[0][1]);
  mma16816<false>(s1, l.p[1], b.p[0][0], b.p[0][1]);
  mma16816<false>(s0, l.p[1], b.p[1][0], b.p[1][1]);
#pragma unroll
  for (int e = 0; e < 4; ++e) o[e] = m[e] + (s1[e] + s0[e]);
}
// sum_{j <= t} coef[t][j] x_j for this lane's tokens t = t0 + 2 (lane % 4) + {0, 1} and both rows of its tiles, where an infinity or a NaN
// among the x must not reach the tokens in front of it (whose coefficients are zeros).
__device__ __noinline__ float4 causal_sum(const float4 x0, const float4 x1, const float* coef, int ld, int t0) {
  const int lane = threadIdx.x & 31, t = t0 + 2 * (lane & 3);
  const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
  float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < CT; ++j) {
    const int from = (lane & ~3) | ((j & 7) >> 1);
    const float a = __shfl_sync(0xffffffffu, x[4 * (j >> 3) + (j & 1)], from), b = __shfl_sync(0xffffffffu, x[4 * (j >> 3) + 2 + (j & 1)], from);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (j <= t + i) {
        const float f = coef[(t + i) * ld + j];
        o[i] = fmaf(f, a, o[i]);
        o[2 + i] = fmaf(f, b, o[2 + i]);
      }
  }
  return make_float4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ bool any_not_finite(const float (&x)[2][4]) {
  float z = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) z = fmaf(x[0][i], 0.f, fmaf(x[1][i], 0.f, z));
  return __any_sync(0xffffffffu, z != 0.f);          // (a NaN is not equal to 0)
}

// A warp's part of the state: columns col, col + 8 (of the block's, by lane), rows 8 i + 2 (lane % 4) + {0, 1} of its share.
template <int NT>
__device__ __forceinline__ void load_state(float (&S)[NT][4], const float* Sg, int V, int row0, int col, int lane) {
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = row0 + 8 * i + 2 * (lane & 3) + (e & 1), j = col + 8 * (e >> 1);
      S[i][e] = j < V ? Sg[(size_t)d * V + j] : 0.f;
    }
}
template <int NT>
__device__ __forceinline__ void store_state(const float (&S)[NT][4], float* Sg, int V, int row0, int col, int lane) {
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = row0 + 8 * i + 2 * (lane & 3) + (e & 1), j = col + 8 * (e >> 1);
      if (j < V) Sg[(size_t)d * V + j] = S[i][e];
    }
}
// (k or q).S over this warp's rows of S: `tile` their part 0, first token.
template <int NK>
__device__ __forceinline__ void state_product(Sums& s0, Sums& s1, const Left (&st)[NK], const __nv_bfloat16* tile, int lane) {
  uint32_t r[2][3][4];
  right_of<false>(r[0], tile, OPROW, lane);
#pragma unroll
  for (int i = 0; i < NK; ++i) {
    if (i + 1 < NK) right_of<false>(r[(i + 1) & 1], tile + 16 * (i + 1), OPROW, lane);
    if (i == 0) six_by_two<true>(s0, s1, st[i], r[i & 1]);
    else six_by_two<false>(s0, s1, st[i], r[i & 1]);
  }
}
// S <- scale S + k^T u over the chunk's tokens, two tiles of rows at a time; scale(i): the factors of tile i's rows of this lane; `tile`: as above.
// The parts of the new S, for the chunk behind, are made while the next tiles' products run.
template <int NT, int NK, typename Scale>
__device__ __forceinline__ void update_state(float (&S)[NT][4], Left (&st)[NK], const Left& u, const __nv_bfloat16* tile, int lane, Scale scale) {
  uint32_t r[2][3][4];
#pragma unroll
  for (int i = 0; i < NT; i += 2) {
    if (i == 0) right_of<true>(r[0], tile, OPROW, lane);
    if (i + 2 < NT) right_of<true>(r[(i / 2 + 1) & 1], tile + 8 * (i + 2), OPROW, lane);
    Sums s0, s1;
    six_by_two<true>(s0, s1, u, r[(i / 2) & 1]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 f = fma2(make_float2(S[i][2 * e], S[i][2 * e + 1]), scale(i), s0.two(e));
      const float2 g = fma2(make_float2(S[i + 1][2 * e], S[i + 1][2 * e + 1]), scale(i + 1), s1.two(e));
      S[i][2 * e] = f.x; S[i][2 * e + 1] = f.y;
      S[i + 1][2 * e] = g.x; S[i + 1][2 * e + 1] = g.y;
    }
    left_of(st[i / 2], S[i], S[i + 1]);
  }
}
__device__ __forceinline__ void group_sync(int group, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(2 + group), "r"(threads) : "memory"); }
__device__ __forceinline__ void loaders_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CLOAD) : "memory"); }

__device__ __forceinline__ void copy16(void* dst, const void* src, bool in) {      // zeros where there is nothing to read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// The chunk of CT tokens that block `x` of a grid over all sequences' chunks looks after: first token and end of the sequence; false: none.
template <int CT>
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

// Block (chunk, key head): a thread per product of two of the chunk's tokens (q_i.k_j for j <= i, k_i.k_j else), then, eight heads
// that share them at a time, a thread per head and column of A, P and T.  (A thread per entry that multiplied its own decays took 40 us
// for 2,048 tokens, 8 key heads and 32 heads: 25 now.)
// (No early start for the kernel behind: its blocks want an SM each, and would be packed in pairs beside this kernel's.)
__global__ void __launch_bounds__(CT * CT, 4) delta_coef_kernel(DeltaArgs a, float* __restrict__ coef, IertBatchView b) {
  constexpr int HEADS = 8;
  __shared__ __align__(16) float k_s[CT][DIM + 4], q_s[CT][DIM + 4], A_s[HEADS][CT][CT];
  __shared__ float dot_s[CT][CT + 1], g_s[HEADS][CT], beta_s[HEADS][CT];
  pdl_wait();
  int tc, t1;
  if (!chunk_of<CT>(b, blockIdx.x, tc, t1)) return;
  const int g = blockIdx.y, GD = a.G * DIM, C = 2 * GD + a.H * a.V, n = min(CT, t1 - tc), rep = a.H / a.G;
  for (int x = threadIdx.x; x < CT * DIM / 4; x += CT * CT) {
    const int t = x / (DIM / 4), d = 4 * (x % (DIM / 4));
    const float* row = a.qkv + (size_t)(tc + min(t, n - 1)) * C + g * DIM + d;
    *reinterpret_cast<float4*>(&q_s[t][d]) = *reinterpret_cast<const float4*>(row);
    *reinterpret_cast<float4*>(&k_s[t][d]) = *reinterpret_cast<const float4*>(row + GD);
  }
  const int hh = threadIdx.x / CT, j = threadIdx.x % CT;
  for (int h0 = g * rep; h0 < (g + 1) * rep; h0 += HEADS) {
    const int h = h0 + hh;
    const bool mine = hh < min(HEADS, (g + 1) * rep - h0);
    if (mine) {
      const bool in = j < n;
      beta_s[hh][j] = in ? a.beta[(size_t)(tc + j) * a.H + h] : 0.f;
      g_s[hh][j] = in ? a.decay[(size_t)(tc + j) * a.H + h] : 1.f;
    }
    __syncthreads();
    if (h0 == g * rep) {
      const float* x = j <= hh ? q_s[hh] : k_s[hh];            // (here hh and j are two tokens)
      const float* y = k_s[j];
      float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll 8
      for (int d = 0; d < DIM; d += 4) {
        const float4 u = *reinterpret_cast<const float4*>(x + d), v = *reinterpret_cast<const float4*>(y + d);
        d0 = fmaf(u.x, v.x, d0); d1 = fmaf(u.y, v.y, d1); d2 = fmaf(u.z, v.z, d2); d3 = fmaf(u.w, v.w, d3);
      }
      dot_s[hh][j] = (d0 + d1) + (d2 + d3);
      __syncthreads();
    }
    float* out = coef + ((size_t)tc * a.H + h) * COEF;         // (rows of tokens: a.H * COEF apart)
    const size_t row = (size_t)a.H * COEF;
    if (mine) {
      float ratio = 1.f;                                       // g_(j+1) .. g_i
#pragma unroll
      for (int i = 0; i < CT; ++i) {
        if (i > j) ratio *= g_s[hh][i];
        A_s[hh][j][i] = j < i ? beta_s[hh][i] * (ratio * dot_s[j][i]) : 0.f;
        if (i < n) {
          out[i * row + CT + j] = j <= i ? ratio * dot_s[i][j] : 0.f;
          if (j == 0) out[i * row + 2 * CT + 1] = g_s[hh][0] * ratio;
        }
      }
      if (j < n) {
        out[j * row + 2 * CT] = beta_s[hh][j];
        out[j * row + 2 * CT + 2] = ratio;
      }
      if (j == 0) out[2 * CT + 3] = g_s[hh][0] * ratio;
    }
    __syncthreads();
    if (mine) {                                      // (1 + A) t = the j-th unit vector
      float t[CT];
#pragma unroll
      for (int m = 0; m < CT; ++m) t[m] = m == j ? 1.f : 0.f;
#pragma unroll
      for (int m = 0; m < CT - 1; ++m) {
        float col[CT];
#pragma unroll
        for (int x = (m + 1) / 4 * 4; x < CT; x += 4) *reinterpret_cast<float4*>(col + x) = *reinterpret_cast<const float4*>(&A_s[hh][m][x]);
#pragma unroll
        for (int x = m + 1; x < CT; ++x) t[x] = m >= j ? fmaf(-col[x], t[m], t[x]) : t[x];   // (a token's NaN stays behind it)
      }
#pragma unroll
      for (int m = 0; m < CT; ++m)
        if (m < n) out[m * row + j] = t[m];
    }
    __syncthreads();
  }
}

constexpr int DWORK = 128;           // computing threads: two column groups x two halves of the rows
struct DeltaShared {
  float v[RING][CT][VROW], c[RING][CT][CROW];
  __nv_bfloat16 op[2][2][3][CT][OPROW];              // q, k in three parts
  __nv_bfloat16 tp[2][2][3][CT][TPROW];              // T, P in three parts
  float4 xk[4][2][32], xq[4][32];                    // a warp's half of the sums k.S, q.S for its partner
};

__global__ void __launch_bounds__(DWORK + CLOAD, 1) delta_chunk_kernel(DeltaArgs a, const float* __restrict__ coef, IertBatchView b) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  DeltaShared& sh = *reinterpret_cast<DeltaShared*>(smem_raw);
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * CCOLS;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const int n_chunks = (t1 - t0 + CT - 1) / CT;

  if (threadIdx.x >= DWORK) {
    // ---------------- loaders: q and k through registers, split a chunk ahead; v and the coefficients three chunks ahead ----------------
    constexpr int ITER = CT * (DIM / 4) / CLOAD, STEP = CLOAD / (DIM / 4);      // a thread's rows of q: every STEP-th
    const int lt = threadIdx.x - DWORK, g = head / (a.H / a.G), GD = a.G * DIM, C = 2 * GD + a.H * a.V;
    const int tq = lt / (DIM / 4), dq = 4 * (lt % (DIM / 4)), tv = lt / (CCOLS / 4), ev = 4 * (lt % (CCOLS / 4));
    const bool in_v = c0 + ev < a.V;
    const float* pq = a.qkv + (size_t)(t0 + tq) * C + g * DIM + dq;
    const float* pv = a.qkv + (size_t)(t0 + tv) * C + 2 * GD + (in_v ? head * a.V + c0 + ev : 0);
    const float* pc = coef + ((size_t)t0 * a.H + head) * COEF;
    float4 f[2 * ITER];
    auto fetch = [&](int n) {
      const int left = t1 - (t0 + n * CT);
      const float* x = pq + (size_t)n * CT * C;
#pragma unroll
      for (int it = 0; it < ITER; ++it) {
        const bool in = tq + it * STEP < left;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        f[it] = in ? *reinterpret_cast<const float4*>(x + (size_t)(it * STEP) * C) : z;
        f[ITER + it] = in ? *reinterpret_cast<const float4*>(x + (size_t)(it * STEP) * C + GD) : z;
      }
    };
    auto ask = [&](int n) {
      if (n < n_chunks) {
        const int left = t1 - (t0 + n * CT), buf = n % RING;
        copy16(&sh.v[buf][tv][ev], tv < left ? pv + (size_t)n * CT * C : a.qkv, tv < left && in_v);
        for (int y = lt; y < CT * COEF / 4; y += CLOAD) {
          const int t = y / (COEF / 4), e = 4 * (y % (COEF / 4));
          copy16(&sh.c[buf][t][e], t < left ? pc + (size_t)(n * CT + t) * a.H * COEF + e : coef, t < left);
        }
      }
      copies_commit();
    };
    auto put4 = [](const float4& x, __nv_bfloat16* dst, int part) {
      uint2 p[3];
      split2(x.x, x.y, p[0].x, p[1].x, p[2].x);
      split2(x.z, x.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(dst + i * part) = p[i];
    };
    auto split = [&](int n) {
      const int out = n & 1, t = lt / 8, e = 4 * (lt % 8);
      const float4 tp = *reinterpret_cast<const float4*>(&sh.c[n % RING][t][e]);        // T, then P
#pragma unroll
      for (int it = 0; it < 2 * ITER; ++it) put4(f[it], &sh.op[out][it / ITER][0][tq + it % ITER * STEP][dq], CT * OPROW);
      put4(tp, &sh.tp[out][e / CT][0][t][e % CT], CT * TPROW);
    };
    fetch(0);
    for (int n = 0; n < RING - 1; ++n) ask(n);
    copies_wait<RING - 2>();
    loaders_sync();                      // every loader's copies of chunk 0
    split(0);
    fetch(1);
    __syncthreads();
    for (int n = 0; n < n_chunks; ++n) {
      copies_wait<RING - 3>();           // chunk n + 1 has arrived ...
      loaders_sync();                    // ... for all loaders
      if (n + 1 < n_chunks) split(n + 1);
      fetch(n + 2);                      // (beyond the last chunk: nothing)
      ask(n + RING - 1);                 // its place was read by the workers before the last barrier
      __syncthreads();
    }
    return;
  }

  // ---------------- workers: warp = (16 columns, half of the rows) ----------------
  constexpr int HROWS = DIM / 2, NT = HROWS / 8, NK = HROWS / 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = warp >> 1, half = warp & 1, q4 = lane & 3, r8 = lane >> 2;
  const int row0 = half * HROWS, col_s = group * 16 + r8, col = c0 + col_s, tok = 8 * half + 2 * q4;
  float* Sg = a.state + (size_t)slot * a.state_stride + a.s_off + (size_t)head * DIM * a.V;
  float* out = a.o + (size_t)(t0 + tok) * a.H * a.V + (size_t)head * a.V + col;
  float S[NT][4];
  Left st[NK];
  load_state(S, Sg, a.V, row0, col, lane);
#pragma unroll
  for (int i = 0; i < NK; ++i) left_of(st[i], S[2 * i], S[2 * i + 1]);
  __syncthreads();
  for (int n = 0; n < n_chunks; ++n) {
    const int buf = n & 1, ring = n % RING;
    const __nv_bfloat16* qo = &sh.op[buf][0][0][0][row0];
    const __nv_bfloat16* ko = &sh.op[buf][1][0][0][row0];
    const float(*co)[CROW] = sh.c[ring];
    // tokens 8 i + 2 q4 + {0, 1} are this lane's: v, beta and G, the weight in the next S
    float v[2][4], from[2][2];
    float2 bg[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = 8 * i + 2 * q4 + h;
        bg[i][h] = *reinterpret_cast<const float2*>(&co[t][2 * CT]);
        from[i][h] = co[t][2 * CT + 2];
        v[i][h] = sh.v[ring][t][col_s];
        v[i][2 + h] = sh.v[ring][t][col_s + 8];
      }
    const float G16 = co[0][2 * CT + 3];
    Sums k0, k1, q0, q1;
    state_product(k0, k1, st, ko, lane);
    Rows T0, T1, P;
    rows_of(T0, &sh.tp[buf][0][0][0][0], lane);
    rows_of(T1, &sh.tp[buf][0][0][8][0], lane);
    rows_of(P, &sh.tp[buf][1][0][8 * half][0], lane);
    float x[2][4];
    k0.all(x[0]);
    k1.all(x[1]);
    sh.xk[warp][0][lane] = make_float4(x[0][0], x[0][1], x[0][2], x[0][3]);
    sh.xk[warp][1][lane] = make_float4(x[1][0], x[1][1], x[1][2], x[1][3]);
    state_product(q0, q1, st, qo, lane);
    group_sync(group, DWORK / 2);
    // x = beta (v - G k.S)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 o = sh.xk[warp ^ 1][i][lane];
      const float p[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i][e] = bg[i][e & 1].x * fmaf(-bg[i][e & 1].y, x[i][e] + p[e], v[i][e]);
    }
    float u[2][4], w[2][4];
    Left l;
    left_of(l, x[0], x[1]);
    six_of_rows(u[0], l, T0);
    six_of_rows(u[1], l, T1);
    // S <- G_16 S + k^T (G_16 / G_j) u_j
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) w[i][e] = u[i][e] * from[i][e & 1];
    left_of(l, w[0], w[1]);
    update_state(S, st, l, ko, lane, [G16](int) { return make_float2(G16, G16); });
    // o = G q.S + P u
    float own[4], other[4], o[4];        // this half of q.S for the eight tokens whose read-out this warp ends with, and for the partner's
    if (half) { q1.all(own); q0.all(other); }
    else { q0.all(own); q1.all(other); }
    sh.xq[warp][lane] = make_float4(other[0], other[1], other[2], other[3]);
    left_of(l, u[0], u[1]);
    six_of_rows(o, l, P);
    if (any_not_finite(u)) {             // (where x has one, u of the tokens in front of it is lost in the product with T too)
      const float4 x0 = make_float4(x[0][0], x[0][1], x[0][2], x[0][3]), x1 = make_float4(x[1][0], x[1][1], x[1][2], x[1][3]);
      const float4 u0 = causal_sum(x0, x1, &co[0][0], CROW, 0), u1 = causal_sum(x0, x1, &co[0][0], CROW, 8);
      const float4 f = causal_sum(u0, u1, &co[0][CT], CROW, 8 * half);
      o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
    }
    group_sync(group, DWORK / 2);
    const float4 f = sh.xq[warp ^ 1][lane];
    const float p[4] = {f.x, f.y, f.z, f.w};
    const int left = t1 - (t0 + n * CT) - tok;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float G = half ? bg[1][e & 1].y : bg[0][e & 1].y;
      if ((e & 1) < left && col + 8 * (e >> 1) < a.V) out[(size_t)(e & 1) * a.H * a.V + 8 * (e >> 1)] = fmaf(G, own[e] + p[e], o[e]);
    }
    out += (size_t)CT * a.H * a.V;
    __syncthreads();
  }
  store_state(S, Sg, a.V, row0, col, lane);
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

#if DIM == 64
// Prompts of 48 tokens a sequence and more, sixteen at a time, as for the delta rule above.  With W_i = w_1 .. w_i (per row of S) the state in front of the
// chunk S gives
//   o_i = (W_(i-1) r_i).S + sum_{j < i} (sum_d r_i k_j w_(j+1) .. w_(i-1)) v_j + (r_i.(u k_i)) v_i
//   S  <- W_16 S + sum_j (w_(j+1) .. w_16 k_j) v_j^T
// There is no chain inside a chunk at all.  The products of two tokens come from a kernel in front with a block per chunk and head;
// here the loaders bring the rows through a ring, scale them by the decays between (products, never quotients) and split them.
// 2,048 tokens, 64 heads of 64 x 64 (128 blocks): 109 us, and 28 of the kernel in front; eight tokens at a time with FFMA 252 in all.

// pairs[token][head][16]: row i of the chunk's products with the tokens j <= i.  Thread (half of the chunk, row d of S): row d's share
// of the pairs inside a half, then summed over the rows; the pairs across the halves are products of r_i w_8 .. w_(i-1) with
// k_j w_(j+1) .. w_7, a dot product of 64 by each of 64 threads.
__global__ void __launch_bounds__(2 * DIM) wkv_pairs_kernel(WkvArgs a, float* __restrict__ pairs, IertBatchView b) {
  constexpr int HT = CT / 2;
  __shared__ float sum_s[2][DIM / 32][36];
  __shared__ __align__(16) float x_s[2][HT][DIM + 4];
  pdl_wait();                                                    // (no early start for the kernel behind, as above)
  int tc, t1;
  if (!chunk_of<CT>(b, blockIdx.x, tc, t1)) return;
  const int head = blockIdx.y, side = threadIdx.x / DIM, d = threadIdx.x % DIM, lane = d & 31, HD = a.H * DIM, n = min(CT, t1 - tc);
  const float bonus = a.u[head * DIM + d];
  float r[HT], k[HT], w[HT];
#pragma unroll
  for (int t = 0; t < HT; ++t) {
    const size_t tok = tc + min(side * HT + t, n - 1);
    const float* row = a.x + tok * a.ld + head * DIM + d;
    r[t] = row[0];
    k[t] = row[HD];
    w[t] = a.decay[tok * HD + head * DIM + d];
  }
  if (side == 0) {
    float e = 1.f;
#pragma unroll
    for (int t = HT - 1; t >= 0; --t) { x_s[0][t][d] = k[t] * e; e *= w[t]; }
  } else {
    float e = 1.f;
#pragma unroll
    for (int t = 0; t < HT; ++t) { x_s[1][t][d] = r[t] * e; e *= w[t]; }
  }
  float p[36];                                                   // pair (i, j <= i) at i (i + 1) / 2 + j
#pragma unroll
  for (int j = 0; j < HT; ++j) {
    p[j * (j + 1) / 2 + j] = r[j] * (bonus * k[j]);
    float e = k[j];
#pragma unroll
    for (int i = j + 1; i < HT; ++i) {
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
  sum_s[side][d / 32][lane] = p[0];
  if (lane < 4) sum_s[side][d / 32][32 + lane] = lane == 0 ? p[32] : lane == 1 ? p[33] : lane == 2 ? p[34] : p[35];
  __syncthreads();
  // (64 threads: the entries across the halves, and zeros behind the diagonal; 64: those of both halves)
  const int i = d / HT, j = d % HT;
  float* row = pairs + ((size_t)(tc + i) * a.H + head) * CT + j;
  const size_t half_on = (size_t)HT * a.H * CT;
  if (side == 0) {
    float t0 = 0.f, t1_ = 0.f;
#pragma unroll
    for (int x = 0; x < DIM; x += 4) {
      const float4 u = *reinterpret_cast<const float4*>(&x_s[1][i][x]), v = *reinterpret_cast<const float4*>(&x_s[0][j][x]);
      t0 = fmaf(u.x, v.x, t0); t1_ = fmaf(u.y, v.y, t1_); t0 = fmaf(u.z, v.z, t0); t1_ = fmaf(u.w, v.w, t1_);
    }
    if (HT + i < n) row[half_on] = t0 + t1_;
    if (i < n) row[HT] = 0.f;
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (h * HT + i < n) {
        float t = 0.f;
        if (j <= i) {
          t = sum_s[h][0][i * (i + 1) / 2 + j];
#pragma unroll
          for (int x = 1; x < DIM / 32; ++x) t += sum_s[h][x][i * (i + 1) / 2 + j];
        }
        row[h * (half_on + HT)] = t;
      }
  }
}

// What the four warps of a column group bring to a sum, added in an order that is the same for all four.
__device__ __forceinline__ void sum_of_four(float (&o)[4], const float4 (*x)[2][32], int part, int tile, int lane) {
  const float4 a = x[part ^ 1][tile][lane], b = x[part ^ 2][tile][lane], c = x[part ^ 3][tile][lane];
  o[0] = (o[0] + a.x) + (b.x + c.x); o[1] = (o[1] + a.y) + (b.y + c.y);
  o[2] = (o[2] + a.z) + (b.z + c.z); o[3] = (o[3] + a.w) + (b.w + c.w);
}

constexpr int PROW = 20, WWORK = 256;           // computing threads: two column groups x four quarters of the rows
struct WkvShared {
  float raw[RING][3][CT][DIM];                       // r, k, w as they are in memory
  float v[RING][CT][VROW], p[RING][CT][PROW];
  __nv_bfloat16 op[2][2][3][CT][OPROW];              // scaled r, k in three parts
  __nv_bfloat16 tp[2][3][CT][TPROW];                 // the products of tokens in three parts
  float wc[2][DIM];
  float4 xo[8][2][32];                               // a warp's share of r.S
};

// PER_SM: blocks that share an SM (80 registers a thread with two, each then slower: 139 us for the one prompt above).  Two are for more blocks than
// two waves of one an SM; this kernel and the one in front, two / one, us: 152 blocks (2,048 tokens of 76 heads) 271 / 248, 256 (two prompts of 1,024, 64
// heads) 156 / 149, 384 (three of 100) 41.8 / 43.8, 1,024 (eight of 48) 45.5 / 52.4.
template <int PER_SM>
__global__ void __launch_bounds__(WWORK + CLOAD, PER_SM) wkv_chunk_kernel(WkvArgs a, const float* __restrict__ pairs, IertBatchView b) {
  static_assert(DIM == 64 && CLOAD == 128, "a loader warp per 64 rows of r or k and half of the tokens");
  extern __shared__ __align__(16) uint8_t smem_raw[];
  WkvShared& sh = *reinterpret_cast<WkvShared*>(smem_raw);
  pdl_wait();
  const int s = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * CCOLS;
  const int slot = b.slot_ids[s];
  const int t0 = b.cu_q[s], t1 = b.cu_q[s + 1];
  if (slot < 0 || t1 <= t0) return;
  const int n_chunks = (t1 - t0 + CT - 1) / CT, HD = a.H * DIM;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x >= WWORK) {
    // ---------------- loaders: three chunks ahead; a warp scales eight tokens of r or of k, a lane two rows of S ----------------
    constexpr int HT = CT / 2, ITER = CT * (DIM / 4) / CLOAD, STEP = CLOAD / (DIM / 4);
    const int lt = threadIdx.x - WWORK;
    const int tq = lt / (DIM / 4), dq = 4 * (lt % (DIM / 4)), tv = lt / (CCOLS / 4), ev = 4 * (lt % (CCOLS / 4)), tp = lt / 4, ep = 4 * (lt % 4);
    const bool in_v = c0 + ev < a.V, of_k = (lt >> 5) & 1;
    const int first = (lt >> 6) * HT, d = 2 * lane;              // this warp's tokens, this lane's rows
    const bool both = first == (of_k ? 0 : HT);                  // the decays of the other half come first
    const float* px = a.x + (size_t)(t0 + tq) * a.ld + head * DIM + dq;
    const float* pw = a.decay + (size_t)(t0 + tq) * HD + head * DIM + dq;
    const float* pv = a.x + (size_t)(t0 + tv) * a.ld + 2 * HD + (in_v ? head * a.V + c0 + ev : 0);
    const float* pp = pairs + ((size_t)(t0 + tp) * a.H + head) * CT + ep;
    auto ask = [&](int n) {
      if (n < n_chunks) {
        const int left = t1 - (t0 + n * CT), buf = n % RING;
        const float* x = px + (size_t)n * CT * a.ld;
        const float* w = pw + (size_t)n * CT * HD;
#pragma unroll
        for (int it = 0; it < ITER; ++it) {
          const int t = tq + it * STEP;
          const bool in = t < left;
          const float* row = in ? x + (size_t)(it * STEP) * a.ld : a.x;
          copy16(&sh.raw[buf][0][t][dq], row, in);
          copy16(&sh.raw[buf][1][t][dq], in ? row + HD : row, in);
          copy16(&sh.raw[buf][2][t][dq], in ? w + (size_t)(it * STEP) * HD : a.decay, in);
        }
        copy16(&sh.v[buf][tv][ev], tv < left ? pv + (size_t)n * CT * a.ld : a.x, tv < left && in_v);
        if (tp < CT) copy16(&sh.p[buf][tp][ep], tp < left ? pp + (size_t)n * CT * a.H * CT : pairs, tp < left);
      }
      copies_commit();
    };
    auto scale = [&](int n) {                                    // a token beyond the sequence: zeros, decay 1
      const int buf = n % RING, out = n & 1, left = t1 - (t0 + n * CT);
      // in the order in which the decays are multiplied: from the first token on for r, from the last one back for k
      auto token = [&](int half, int i) { return half + (of_k ? HT - 1 - i : i); };
      auto decay = [&](int t) { return t < left ? *reinterpret_cast<const float2*>(&sh.raw[buf][2][t][d]) : make_float2(1.f, 1.f); };
      float2 f = make_float2(1.f, 1.f), x[HT], w[HT];            // (every load before the first store: they would wait for one another)
#pragma unroll
      for (int i = 0; i < HT; ++i) {
        x[i] = *reinterpret_cast<const float2*>(&sh.raw[buf][of_k][token(first, i)][d]);
        w[i] = decay(token(first, i));
      }
      if (both) {
#pragma unroll
        for (int i = 0; i < HT; ++i) f = mul2(f, decay(token(HT - first, i)));
      }
      const float4 y = *reinterpret_cast<const float4*>(&sh.p[buf][tp % CT][ep]);
#pragma unroll
      for (int i = 0; i < HT; ++i) {
        const float2 z = mul2(x[i], f);
        f = mul2(f, w[i]);
        uint32_t p[3];
        split2(z.x, z.y, p[0], p[1], p[2]);
#pragma unroll
        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint32_t*>(&sh.op[out][of_k][m][token(first, i)][d]) = p[m];
      }
      if (both && !of_k) *reinterpret_cast<float2*>(&sh.wc[out][d]) = f;
      if (tp < CT) {
        uint2 p[3];
        split2(y.x, y.y, p[0].x, p[1].x, p[2].x);
        split2(y.z, y.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint2*>(&sh.tp[out][m][tp][ep]) = p[m];
      }
    };
    for (int n = 0; n < RING - 1; ++n) ask(n);
    copies_wait<RING - 2>();
    loaders_sync();                      // every loader's copies of chunk 0
    scale(0);
    __syncthreads();
    for (int n = 0; n < n_chunks; ++n) {
      copies_wait<RING - 3>();           // chunk n + 1 has arrived ...
      loaders_sync();                    // ... for all loaders
      if (n + 1 < n_chunks) scale(n + 1);
      ask(n + RING - 1);                 // its place: read by the workers before the last barrier, scaled from two chunks ago
      __syncthreads();
    }
    return;
  }

  // ---------------- workers: warp = (16 columns, a quarter of the rows) ----------------
  constexpr int QROWS = DIM / 4, NT = QROWS / 8, NK = QROWS / 16;
  const int warp = threadIdx.x >> 5, group = warp >> 2, part = warp & 3, q4 = lane & 3, r8 = lane >> 2;
  const int row0 = part * QROWS, col_s = group * 16 + r8, col = c0 + col_s;
  const bool reads = part < 2;           // two of the four read out, eight tokens each
  const int tok = 8 * part + 2 * q4;
  float* Sg = a.state + (size_t)slot * a.state_stride + a.s_off + (size_t)head * DIM * a.V;
  float* out = a.o + (size_t)(t0 + tok) * a.H * a.V + (size_t)head * a.V + col;
  float S[NT][4];
  Left st[NK];
  load_state(S, Sg, a.V, row0, col, lane);
#pragma unroll
  for (int i = 0; i < NK; ++i) left_of(st[i], S[2 * i], S[2 * i + 1]);
  __syncthreads();
  for (int n = 0; n < n_chunks; ++n) {
    const int buf = n & 1, ring = n % RING;
    float v[2][4], y[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) v[i][e] = sh.v[ring][8 * i + 2 * q4 + (e & 1)][col_s + 8 * (e >> 1)];
    {
      Sums s0, s1;
      state_product(s0, s1, st, &sh.op[buf][0][0][0][row0], lane);
      s0.all(y[0]);
      s1.all(y[1]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (i != part) sh.xo[warp][i][lane] = make_float4(y[i][0], y[i][1], y[i][2], y[i][3]);
    }
    Left vl;
    left_of(vl, v[0], v[1]);
    const float* wc = &sh.wc[buf][row0 + 2 * q4];
    update_state(S, st, vl, &sh.op[buf][1][0][0][row0], lane, [wc](int i) { return *reinterpret_cast<const float2*>(wc + 8 * i); });
    group_sync(group, WWORK / 2);
    if (reads) {
      Rows P;
      rows_of(P, &sh.tp[buf][0][8 * part][0], lane);
      float o[4], rs[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) rs[e] = part ? y[1][e] : y[0][e];
      sum_of_four(rs, sh.xo + 4 * group, part, part, lane);
      six_of_rows(o, vl, P);
      if (any_not_finite(v)) {
        const float4 f = causal_sum(make_float4(v[0][0], v[0][1], v[0][2], v[0][3]), make_float4(v[1][0], v[1][1], v[1][2], v[1][3]), &sh.p[ring][0][0], PROW, 8 * part);
        o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
      }
      const int left = t1 - (t0 + n * CT) - tok;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if ((e & 1) < left && col + 8 * (e >> 1) < a.V) out[(size_t)(e & 1) * a.H * a.V + 8 * (e >> 1)] = rs[e] + o[e];
      out += (size_t)CT * a.H * a.V;
    }
    __syncthreads();
  }
  store_state(S, Sg, a.V, row0, col, lane);
}

// The same for sequences of few tokens, eight at a time with FFMA: a thread owns DIM / 16 rows of four columns of S, two rows an instruction, and the
// sums of a token over the 16 lanes of a column are added together.  Such a step is many short chains, which want many small blocks on
// an SM and little padding (layers at 4,096, eight / sixteen at a time, us: 128 sequences of 8 tokens 476 / 561, of 16 707 / 776, of 32 1,207 / 1,250;
// 16 sequences of 24 262 / 270, of 48 306 / 305; 4 of 128 275 / 273, one of 2,048 688 / 570).
namespace eight {
constexpr int CT = 8, CG = 4, CL = 16, CWORK = 128, CCOLS = CWORK / CL * CG;
constexpr int CP = DIM / CL / 2;                              // pairs of rows per lane

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

constexpr int WLOAD = DIM;

// pairs[token][head][8]: row i of the chunk's products with the tokens j <= i.  Thread d: row d's share, then summed over the rows.
__global__ void __launch_bounds__(DIM) wkv_pairs_kernel(WkvArgs a, float* __restrict__ pairs, IertBatchView b) {
  __shared__ float sum_s[DIM / 32][36];
  pdl_wait();                                                    // (no early start for the kernel behind, as for the delta rule)
  int tc, t1;
  if (!chunk_of<CT>(b, blockIdx.x, tc, t1)) return;
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
}  // namespace eight
#endif

// Lanes per column: the fewest that give the device about eight warps per SM (at most 32), and columns per
// CTA so that a CTA has up to 256 computing threads.  (Measured at 32 heads of 128 x 128, one prompt of 2,048
// tokens: 8 lanes per column 1.08 ms, 16 lanes 0.91 ms, 32 lanes 1.42 ms per layer.)
#if IERT_CHUNKED
// Prompts go sixteen (eight) tokens at a time; steps of few tokens per sequence token after token: a chunk costs what all its tokens cost, the
// kernel in front is one launch more, and such a step is bound by reading and writing the state.  Where the line lies (layers at 4,096, sequences of
// equal length, chunks / token after token, us):
//   delta rule, 16 tokens a sequence: two sequences 75 / 78, four 87 / 90, 16 188 / 206, 64 430 / 515, 128 797 / 986; 17 tokens 79 / 80, 102 / 98,
//   198 / 198, 546 / 557, 1,003 / 1,011; one sequence of 17 70 / 67, of 24 71 / 70, of 32 73 / 75, of 128 104 / 131; 64 tokens 106 / 135, 165 / 190,
//   318 / 418, 1,062 / 1,455;
//   decays per channel (eight at a time): one sequence of 4 to 32 tokens 71 / 70 to 109 / 110, two of 8 82 / 81, four of 8 110 / 113, eight of
//   4 114 / 118 and of 16 138 / 165, 32 of 4 170 / 185.
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

// Scratch (floats) of the recurrences over n_tokens tokens and H heads: the products of tokens with one another, for the delta rule with what
// else its chunks need; for the decay per key channel a row of products alone.
IERT_API long long iert_recurrent_scratch_floats(int n_tokens, int H) { return (long long)n_tokens * H * 36; }
IERT_API long long iert_wkv_scratch_floats(int n_tokens, int H) { return (long long)n_tokens * H * 16; }      // (eight of them: chunks of eight tokens)

// scratch: as many floats as above, or null (then tokens go one after another)
IERT_API int iert_delta_recur(const float* qkv, const float* beta, const float* decay, float* state,
                              long long state_stride, long long s_off, float* o, float* scratch, int G, int H, int V,
                              const IertBatchView* batch, cudaStream_t stream) {
  if (batch->n_seqs <= 0 || batch->n_tokens <= 0) return IERT_OK;
  if (G <= 0 || H <= 0 || H % G || V <= 0 || H > 65535) return IERT_BAD_ARGUMENT;
#if IERT_CHUNKED
  if (scratch && chunked(batch, 16, 32) && V % 4 == 0 && (2 * G * DIM + H * V) % 4 == 0 && state_stride % 4 == 0 && s_off % 4 == 0 &&
      (((uintptr_t)qkv | (uintptr_t)state | (uintptr_t)o | (uintptr_t)scratch) & 15) == 0) {
    DeltaArgs a = {qkv, beta, decay, state, state_stride, s_off, o, G, H, V, CCOLS};
    if (cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DeltaShared)) != cudaSuccess)
      return iert_check_launch("delta_recur attribute");
    launch_dep(delta_coef_kernel, dim3(batch->n_tokens / CT + batch->n_seqs, G), dim3(CT * CT), 0, stream, a, scratch, *batch);
    launch_dep(delta_chunk_kernel, dim3(batch->n_seqs, H, (V + CCOLS - 1) / CCOLS), dim3(DWORK + CLOAD), sizeof(DeltaShared), stream, a,
               (const float*)scratch, *batch);
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
    const dim3 columns(batch->n_seqs, H, (V + CCOLS - 1) / CCOLS);
    if (chunked(batch, 48, 48)) {
      auto* kernel = (long long)columns.x * columns.y * columns.z > 2 * iert_sm_count_cached() ? wkv_chunk_kernel<2> : wkv_chunk_kernel<1>;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WkvShared)) != cudaSuccess)
        return iert_check_launch("wkv_recur attribute");
      launch_dep(wkv_pairs_kernel, dim3(batch->n_tokens / CT + batch->n_seqs, H), dim3(2 * DIM), 0, stream, a, scratch, *batch);
      launch_dep(kernel, columns, dim3(WWORK + CLOAD), sizeof(WkvShared), stream, a, (const float*)scratch, *batch);
    } else {
      static_assert(eight::CCOLS == CCOLS, "the same grid");
      launch_dep(eight::wkv_pairs_kernel, dim3(batch->n_tokens / eight::CT + batch->n_seqs, H), dim3(DIM), 0, stream, a, scratch, *batch);
      launch_dep(eight::wkv_chunk_kernel, columns, dim3(eight::CWORK + eight::WLOAD), 0, stream, a, (const float*)scratch, *batch);
    }
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
