// Projection of a 32-bit run on the tensor cores: out[t, n] = sum_k x[t, k] w[n, k], all fp32, for the inner axes at which
// its error against exact arithmetic is well below that of the one-accumulator fp32 sum of gemm_plain.cu (which stays for what this
// kernel does not take).
//
// An fp32 number is the sum of three bf16 numbers: the nearest one, the nearest to the remainder, and what is left (exactly, unless it
// falls below 2^-133, bf16's smallest number), so x w is the sum of nine bf16 products.  Six are formed on tcgen05; the other three come to
// 2^-24 of the product at most, of either sign.  (Parts cut off instead of rounded left up to 2^-21, always of the product's sign: rows with
// one number among zeros had 2.5 times the plain kernel's error.)  The tensor core adds with a few bits less care than an fp32
// addition, so no sum stays there for long: the products of 64 k are summed in tensor memory and then added to fp32 registers
// by ordinary rounded additions, K / 64 of them per output; the main product (first part times first part) has a tensor-memory
// sum of its own, so that few additions there meet a sum as large as the result.  Relative error (2-norm) against 64 bits, this
// kernel / gemm_plain.cu: K of 1,024: 9.0e-8 / 5.8e-7 (8.9e-8 / 5.0e-7 where all numbers are positive); 4,096: 1.1e-7 / 1.2e-6;
// 14,336: 1.6e-7 / 2.2e-6.  Sums that are short because nearly all of a row is zero have the same error in both: one number in a row
// 2.6e-8 / 2.5e-8, eight 5.5e-8 / 5.3e-8 (with the two next products as well 2.5e-8 and 5.5e-8, and a tenth more time).
//
// Measured (gemm_plain.cu in brackets): 333 tokens x 28,672 x 4,096 0.72 ms (4.43), 333 x 4,096 x 14,336 0.39 ms (2.46), one token
// x 28,672 x 4,096 0.27 ms (0.96), x 4,096 x 14,336 0.12 ms (2.38).  What bounds it is the chain of a block (copy, split, MMAs, read
// back: about 2,000 cycles for 128 tokens); the six products alone are 768.  The weights' parts in tensor memory instead of shared memory (96 tokens
// a tile then) were no faster, 778 us for the first of these, nor tokens split by a kernel in front, 903.  An 8 x 8 register tile of fp32 multiply-adds reached
// 2.1 ms on the first of these sizes: shared memory returns one operand word per lane and cycle, which that tile needs in full.
//
// Roles: TMA brings fp32 tiles of 32 k into a ring; warps 8-15 split them into swizzled operand tiles, two to four blocks deep; warp 16 asks for the
// tiles and issues the 12 MMAs of a block (128 weight rows on the M side, BT tokens on the N side), converged, one lane acting (a lane of
// warp 0 did so between its additions, each MMA's operands moved to uniform registers one by one: 839 us where this takes 742); warps 0-7 add every second
// block's sums (64 k) to their registers while the next one's MMAs run.  A matrix with few rows is split over k between the
// CTAs of a cluster (by the matrix's shape alone, so that a row's result does not depend on how many rows the call has), which
// add their parts in order through distributed shared memory: no scratch, no counters.  An output that is not finite (an
// infinity or NaN among its inputs, or an overflow) is computed again as gemm_plain.cu does, and so is one below 2^-60, whose inputs may
// have lost bits below 2^-133 (a loss of K 2^-134 |w| at most, under 2^-24 of a larger output for weights up to 2^36); a zero, as rows of
// zeros give by the thousand, stays.
#include "common.cuh"
#include "sm100.cuh"

using namespace iert;
using namespace sm100;

namespace {

constexpr int TILE_N = 128, BLOCK_K = 32, THREADS = 17 * 32;
constexpr int W_PART_BYTES = TILE_N * BLOCK_K * 2, W_STAGE_BYTES = TILE_N * BLOCK_K * 4;
constexpr uint32_t WAIT_LIMIT = 1u << 22;

struct F32Params {
  const float* x;
  const float* w;
  float* out;
  long long ldx, ldw, ldo;
  int M, N, K, add, t_tiles, splits, kb_total, kb_per_split;
  int* err;
};

__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t addr, int rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}

// Eight fp32 numbers into three 16-byte runs of bf16: every part the nearest to what is left, every remainder exact.
__device__ __forceinline__ void split8(const float4& a, const float4& b, uint4& p0, uint4& p1, uint4& p2) {
  const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t* o0 = reinterpret_cast<uint32_t*>(&p0);
  uint32_t* o1 = reinterpret_cast<uint32_t*>(&p1);
  uint32_t* o2 = reinterpret_cast<uint32_t*>(&p2);
  auto nearest = [](float x, float y) {
    const __nv_bfloat162 two = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&two);
  };
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float x = v[2 * i], y = v[2 * i + 1];
    o0[i] = nearest(x, y);
    const float xr = x - __uint_as_float(o0[i] << 16), yr = y - __uint_as_float(o0[i] & 0xffff0000u);
    o1[i] = nearest(xr, yr);
    o2[i] = nearest(xr - __uint_as_float(o1[i] << 16), yr - __uint_as_float(o1[i] & 0xffff0000u));
  }
}

// gemm_plain.cu's sum: one accumulator, k ascending.
__device__ __noinline__ float plain_dot(const float* x, const float* w, int K) {
  float s = 0.f;
  for (int k = 0; k < K; k += 4) {
    const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
    s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
  }
  return s;
}

__device__ __forceinline__ void put(const F32Params& p, int t, int n, float v) {
  if (t >= p.M || n >= p.N) return;
  if (!isfinite(v) || (v != 0.f && fabsf(v) < 0x1p-60f)) v = plain_dot(p.x + (long long)t * p.ldx, p.w + (long long)n * p.ldw, p.K);
  float* o = p.out + (long long)t * p.ldo + n;
  *o = p.add ? *o + v : v;
}

// Eight consecutive fp32 columns of this thread's TMEM lane (tmem_ld_wait() before they are used).
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// K-major operand tile with rows of 64 bytes (32 bf16) under the 64-byte swizzle: 8-row groups are 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

// Operand buffers (as many as leave room for four blocks of 32 k in the ring in front of the converters, at most four), ring.
template <int BT>
struct Plan {
  static constexpr int STAGE_BYTES = W_STAGE_BYTES + BT * BLOCK_K * 4;
  static constexpr int BUF_BYTES = 3 * (W_PART_BYTES + BT * BLOCK_K * 2);
  static constexpr int ROOM = 222 * 1024;
  static constexpr int BUFS = BT <= 32 ? 4 : BT <= 64 ? 3 : 2;
  static constexpr int FIT = (ROOM - BUFS * BUF_BYTES) / STAGE_BYTES;
  static constexpr int STAGES = FIT > 8 ? 8 : FIT;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + BUFS * BUF_BYTES + 1024;
};

template <int BT>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                 const __grid_constant__ CUtensorMap map_x, const F32Params p) {
  using P = Plan<BT>;
  constexpr int X_PART_BYTES = BT * BLOCK_K * 2;
  // two buffers of (small products, main products)
  constexpr uint32_t ACC_COLS = BT <= 16 ? 64 : BT <= 32 ? 128 : BT <= 64 ? 256 : 512;
  constexpr uint32_t IDESC = instr_desc_bf16(TILE_N, BT);
  constexpr int W_ITEMS = TILE_N / 64, X_ITEMS = (BT + 63) / 64;     // rows a converter thread looks after
  constexpr int CPT = BT / 2;                                                 // outputs of an accumulating thread
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = smem + P::BUFS * P::BUF_BYTES;                                 // behind the operand buffers
  __shared__ uint64_t st_full[P::STAGES], op_full[P::BUFS], op_empty[P::BUFS], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x % p.splits, tile = blockIdx.x / p.splits;      // the CTAs of a cluster are one tile's splits
  const int n0 = (tile / p.t_tiles) * TILE_N, t0 = (tile % p.t_tiles) * BT;
  const int kb0 = split * p.kb_per_split, n_kb = max(0, min(p.kb_total - kb0, p.kb_per_split));
  if (threadIdx.x == 0) {
    for (int i = 0; i < P::STAGES; ++i) mbar_init(&st_full[i], 1);
    for (int i = 0; i < P::BUFS; ++i) { mbar_init(&op_full[i], 8); mbar_init(&op_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 8);
    }
    abort_s = 0;
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(&tmem_slot, ACC_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  if (threadIdx.x == 0) pdl_launch_dependents();
  float* part = reinterpret_cast<float*>(smem);      // [BT][TILE_N], where the operands were: this split's sums
  bool ok = true;

  auto load_w = [&](int b) {
    const int s = b % P::STAGES;
    mbar_expect_tx(&st_full[s], P::STAGE_BYTES);
    tma_load_2d(ring + s * P::STAGE_BYTES, &map_w, &st_full[s], (kb0 + b) * BLOCK_K, n0);
  };
  auto load_x = [&](int b) {
    const int s = b % P::STAGES;
    tma_load_2d(ring + s * P::STAGE_BYTES + W_STAGE_BYTES, &map_x, &st_full[s], (kb0 + b) * BLOCK_K, t0);
  };

  if (warp == 16) {
    // ---------------- tiles and MMAs ----------------
    const uint32_t leader = elect_leader();
    int asked = min(n_kb, P::STAGES);
    if (lane == 0) {
      tma_prefetch_desc(&map_w);
      tma_prefetch_desc(&map_x);
      for (int b = 0; b < asked; ++b) load_w(b);                               // the weights do not depend on the kernel in front
      pdl_wait();
      for (int b = 0; b < asked; ++b) load_x(b);
    }
    __syncwarp();
    // a wait of the whole warp: what one lane sees, all act on
    auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag)) != 0; };
    int buf = 0;
    uint32_t o_phase = 0;
    for (int q = 0; ok && 2 * q < n_kb; ++q) {
      // the MMAs of blocks 2 q and 2 q + 1: the main product x0 w0 in a sum of its own, the five small ones in another
      if (!warp_wait(&acc_empty[q & 1], ((q >> 1) & 1) ^ 1)) { ok = false; break; }
      const uint32_t d = tmem_base + (uint32_t)((q & 1) * 2 * BT);
      for (int b = 2 * q; b < min(2 * q + 2, n_kb); ++b) {
        if (!warp_wait(&op_full[buf], o_phase)) { ok = false; break; }
        if (asked < n_kb) {                                                    // block b has left its place in the ring
          if (lane == 0) { load_w(asked); load_x(asked); }
          ++asked;
          __syncwarp();
        }
        tc_fence_after();
        const uint32_t wa = smem_addr(smem + buf * P::BUF_BYTES), xa = wa + 3 * W_PART_BYTES;
        constexpr int WP[6] = {2, 0, 1, 1, 0, 0}, XP[6] = {0, 2, 1, 0, 1, 0};  // (part of w, part of x)
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          const uint64_t da = smem_desc_k64(wa + WP[m] * W_PART_BYTES), db = smem_desc_k64(xa + XP[m] * X_PART_BYTES);
#pragma unroll
          for (int ks = 0; ks < BLOCK_K / 16; ++ks)
            mma_ss(leader, d + (m == 5 ? BT : 0), da + 2 * ks, db + 2 * ks, IDESC, ((b & 1) || (m != 0 && m != 5) || ks > 0) ? 1u : 0u);
        }
        mma_commit(leader, &op_empty[buf]);
        if (++buf == P::BUFS) { buf = 0; o_phase ^= 1; }
      }
      if (ok) mma_commit(leader, &acc_full[q & 1]);
    }
    if (!ok) {
      *abort_flag = 1;
      if (lane == 0)                                                           // copies under way land before the CTA ends
        for (int b = max(0, asked - P::STAGES); b < asked; ++b) mbar_wait(&st_full[b % P::STAGES], (b / P::STAGES) & 1, WAIT_LIMIT);
    }
  } else if (warp >= 8) {
    // ---------------- converters ----------------
    const int ct = threadIdx.x - 8 * 32, row = ct >> 2, chunk = ct & 3;       // 64 rows x 4 runs of 8 k per pass
    // eight lanes read two rows of 128 bytes: odd rows take their second 16 bytes first, so that no two lanes meet in a bank
    const int half = (row & 1) * 16;
    const uint32_t in_off = row * 128 + chunk * 32;
    const uint32_t out_off = row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
    int s = 0, buf = 0;
    uint32_t s_phase = 0, o_phase = 1;
    for (int b = 0; b < n_kb; ++b) {
      if (!wait_or_abort(&st_full[s], s_phase, abort_flag) || !wait_or_abort(&op_empty[buf], o_phase, abort_flag)) ok = false;
      if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
      const uint8_t* in = ring + s * P::STAGE_BYTES + in_off;
      uint8_t* out = smem + buf * P::BUF_BYTES + out_off;
#pragma unroll
      for (int i = 0; i < W_ITEMS + X_ITEMS; ++i) {
        if (i >= W_ITEMS && BT % 64 && row + 64 * (i - W_ITEMS) >= BT) break;
        const uint8_t* src = in + i * 64 * 128;                                // the tokens' rows follow the weights'
        const float4 u = *reinterpret_cast<const float4*>(src + half), v = *reinterpret_cast<const float4*>(src + (half ^ 16));
        float4 lo, hi;
        lo.x = half ? v.x : u.x; lo.y = half ? v.y : u.y; lo.z = half ? v.z : u.z; lo.w = half ? v.w : u.w;
        hi.x = half ? u.x : v.x; hi.y = half ? u.y : v.y; hi.z = half ? u.z : v.z; hi.w = half ? u.w : v.w;
        uint4 p0, p1, p2;
        split8(lo, hi, p0, p1, p2);
        uint8_t* dst = i < W_ITEMS ? out + i * 64 * 64 : out + 3 * W_PART_BYTES + (i - W_ITEMS) * 64 * 64;
        const int part = i < W_ITEMS ? W_PART_BYTES : X_PART_BYTES;
        *reinterpret_cast<uint4*>(dst) = p0;
        *reinterpret_cast<uint4*>(dst + part) = p1;
        *reinterpret_cast<uint4*>(dst + 2 * part) = p2;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_full[buf]);
      if (++s == P::STAGES) { s = 0; s_phase ^= 1; }
      if (++buf == P::BUFS) { buf = 0; o_phase ^= 1; }
    }
  } else {
    // ---------------- accumulation: warp w reads TMEM lanes 32 (w % 4).., the columns of its half ----------------
    const int n_pairs = (n_kb + 1) / 2;
    float acc[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) acc[j] = 0.f;
    pdl_wait();                                   // (the residual is read and written below)
    const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * CPT);
    for (int q = 0; q < n_pairs; ++q) {
      if (!wait_or_abort(&acc_full[q & 1], (q >> 1) & 1, abort_flag)) ok = false;
      if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
      tc_fence_after();
      const uint32_t src = taddr + (q & 1) * 2 * BT;
      constexpr int STEP = CPT % 16 || CPT == 64 ? 8 : 16;
#pragma unroll
      for (int c = 0; c < CPT; c += STEP) {
        float v[STEP], u[STEP];
        if constexpr (STEP == 16) {
          tmem_ld16_issue(src + c, reinterpret_cast<uint32_t*>(v));
          tmem_ld16_issue(src + BT + c, reinterpret_cast<uint32_t*>(u));
        } else {
          tmem_ld8_issue(src + c, reinterpret_cast<uint32_t*>(v));
          tmem_ld8_issue(src + BT + c, reinterpret_cast<uint32_t*>(u));
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < STEP; ++j) acc[c + j] += v[j] + u[j];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[q & 1]);
    }
    const int n_local = (warp & 3) * 32 + lane, c0 = (warp >> 2) * CPT;
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      if (p.splits == 1) put(p, t0 + c0 + j, n0 + n_local, acc[j]);
      else part[(c0 + j) * TILE_N + n_local] = acc[j];
    }
  }
  if (!ok) {
    atomicOr(p.err, IERT_ERR_WAIT_EXPIRED);
    *abort_flag = 1;
  }
  if (p.splits > 1) {
    __syncwarp();
    cluster_sync();
    // this CTA adds its share of the token rows, the splits in order
    const int rows = BT / p.splits;
    for (int i = threadIdx.x; i < rows * TILE_N; i += THREADS) {
      const int t = split * rows + i / TILE_N, n = i % TILE_N;
      if (t0 + t >= p.M) break;
      const uint32_t a = smem_addr(part + t * TILE_N + n);
      float s = ld_cluster(a, 0);
      for (int r = 1; r < p.splits; ++r) s += ld_cluster(a, r);
      put(p, t0 + t, n0 + n, s);
    }
    __syncwarp();
    cluster_sync();                                                          // nobody leaves while its part is read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ACC_COLS);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// An fp32 row-major matrix [rows, cols] with row stride ld, loaded in boxes of box_rows x 32.
bool tensor_map_f32(const float* ptr, long long rows, long long cols, long long ld, int box_rows, CUtensorMap* out) {
  static EncodeTiledFn fn = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      sym = nullptr;
    return (EncodeTiledFn)sym;
  }();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {(cuuint32_t)BLOCK_K, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  return fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BT>
int launch(const F32Params& p, int tiles, cudaStream_t stream) {
  CUtensorMap mw, mx;
  if (!tensor_map_f32(p.w, p.N, p.K, p.ldw, TILE_N, &mw) || !tensor_map_f32(p.x, p.M, p.K, p.ldx, BT, &mx)) return IERT_BAD_ARGUMENT;
  if (cudaFuncSetAttribute(gemm_f32_tc_kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Plan<BT>::SMEM) != cudaSuccess)
    return iert_check_launch("gemm_f32_tc attribute");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.splits);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = Plan<BT>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = iert_pdl_enabled ? 2 : 1;
  cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel<BT>, mw, mx, p);
  return iert_check_launch("gemm_f32_tc");
}

}  // namespace

// x [M, K], w [N, K], out [M, N], fp32 with row strides ldx, ldw, ldo (elements).  mode 0 stores, 1 adds into out.  Taken: K of
// 1,024 or more (below that the sums are short and the plain kernel's error is the smaller one), K a multiple of 4, rows on
// 16-byte boundaries; otherwise IERT_BAD_ARGUMENT and nothing is launched.
IERT_API int iert_gemm_f32_tc(const float* x, const float* w, float* out, int M, int N, int K, long long ldx, long long ldw,
                              long long ldo, int mode, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return IERT_OK;
  if (K < 1024 || (K & 3) || (ldx & 3) || (ldw & 3) || (((uintptr_t)x | (uintptr_t)w) & 15) || (mode != 0 && mode != 1))
    return IERT_BAD_ARGUMENT;
  F32Params p = {x, w, out, ldx, ldw, ldo, M, N, K, mode, 1, 1, (K + BLOCK_K - 1) / BLOCK_K, 0, err};
  const int n_tiles = (N + TILE_N - 1) / TILE_N;
  // the splits follow from the matrix alone: as many as keep one token tile's CTAs within one per SM
  while (p.splits < 4 && 2 * p.splits * n_tiles <= iert_sm_count_cached() && p.kb_total / (2 * p.splits) >= 8) p.splits *= 2;
  p.kb_per_split = (p.kb_total + p.splits - 1) / p.splits;
  // as few tiles of up to 128 tokens as there can be, of the fewest tokens (a row's result does not depend on the tile: 333 tokens in three of
  // 112 instead of three of 128: x 28,672 x 4,096 742 -> 716 us, x 4,096 x 14,336 405 -> 387)
  const int least = (M + 127) / 128, each = (M + least - 1) / least;
  const int bt = each <= 16 ? 16 : each <= 32 ? 32 : each <= 64 ? 64 : (each + 15) / 16 * 16;
  p.t_tiles = (M + bt - 1) / bt;
  const long long tiles = (long long)n_tiles * p.t_tiles;
  if (tiles * p.splits > 0x7fffffff) return IERT_BAD_ARGUMENT;
  switch (bt) {
    case 16: return launch<16>(p, (int)tiles, stream);
    case 32: return launch<32>(p, (int)tiles, stream);
    case 64: return launch<64>(p, (int)tiles, stream);
    case 80: return launch<80>(p, (int)tiles, stream);
    case 96: return launch<96>(p, (int)tiles, stream);
    case 112: return launch<112>(p, (int)tiles, stream);
    default: return launch<128>(p, (int)tiles, stream);
  }
}
