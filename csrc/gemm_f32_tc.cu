// fp32 GEMM on the tensor cores: operands split into three bf16 parts, products summed as closely as multiply-adds sum them.
//
// An fp32 value is exactly h + m + l with three bf16 parts of 8 significant bits each (rounded to nearest, so m and l may
// carry the other sign).  Of the nine products of two such values six are formed, h h, h m, m h, m m, h l, l h; what is left
// out, m l + l m + l l, is below 2^-25 of the product, less than the rounding of one fp32 multiply.  Every bf16 product is exact; the
// accumulator is not: tcgen05 truncates where an fma rounds, so a long chain drifts towards zero.  Therefore the small
// products of a k-block go first (their truncations are 2^-8 of an ulp), h h last, and after 64 terms the block's sum leaves
// TMEM and is added in fp32 registers, rounded to nearest: four truncated steps, not K / 16, ever meet in one accumulator.
//
// A CTA computes a 128 x BN tile over one part of K.  Its 16 warps do everything: fetch the next k-block from global memory
// into registers, split the present one into shared memory (swizzled bf16 tiles in the operand's own orientation: K-major or
// MN-major descriptors, no transpose), one thread issues the 24 MMAs, and while they run all warps add the block before to
// their registers and split the next.  The parts of K are CTAs of one cluster: each leaves its partial tile in its own shared
// memory and every CTA of the cluster adds an equal share of the rows, in the order of the parts, and runs the epilogue on it.
// Deterministic, and no scratch in global memory.
//
// Bits below 2^-134 do not fit a bf16 part, and a value that is not finite, or rounds to infinity in bf16, makes NaN of its
// parts.  An output that is not finite, or not zero and below 2^-100, is therefore computed once more as one run of fma over K: it
// then is what multiply-adds make of it.
//
// Distance from fp64 (2-norm, relative; B200) against the multiply-add tiles: normal operands, 509 x 768 x 768 0.95e-7 (2.1e-7),
// K = 3072 1.1e-7 (2.9e-7), 256 x 256 x 1024 1.0e-7 (1.6e-7); GELU outputs the same; operands that are all positive, where the
// truncations add up, 0.9e-7 (0.8e-7).
//
// What bounds it: shared memory.  A k-block at BN = 128 writes 96 KB of parts and its MMAs read 192 KB, 2300 clocks at 128 bytes
// each, against 1536 of the MMAs alone; fetching 64 KB ahead of the split only partly overlaps it (4000 clocks measured).  It is
// still 2.4 times the rate of the packed multiply-adds (2048^3: 352 -> 144 us).
#include <atomic>

#include "gemm_f32.cuh"

namespace dptb {

constexpr int kTcBM = 128, kTcBK = kF32TcBK;
constexpr int kTcMaxSplits = 8;                      // CTAs of a cluster
constexpr int kTcThreads = 512;                      // 16 warps that fetch, split and add; one more issues the MMAs

template <int BN>
struct TcF32Smem {
  static constexpr int kAPart = kTcBM * 128, kBPart = BN * 128;     // one bf16 part of a k-block: 128 bytes a row
  static constexpr int kStage = 3 * (kAPart + kBPart);
  static constexpr int kOutLd = BN + 4;                            // floats; 16-byte rows, quarter-warps on different banks
  static constexpr int kBarOff = 2 * kStage;
  static constexpr int kTotal = kBarOff + 64 + 1024;
  static_assert(kTcBM * kOutLd * 4 <= 2 * kStage, "the partial tile reuses the stages");
};

// Chunks of eight neighbouring elements of an operand's k-block, R rows (columns) of M (N) x 64 of K, one 16-byte piece of each part
// per chunk.  MN: the operand's M / N axis is contiguous, else its K axis.
template <int R, bool MN>
struct SplitTile {
  static constexpr int kChunks = R * kTcBK / 8 / kTcThreads;
  static_assert(R * kTcBK / 8 % kTcThreads == 0, "whole chunks per thread");
  float v[kChunks][8];

  static __device__ __forceinline__ void place(int i, int& mn, int& k) {
    const int idx = threadIdx.x + i * kTcThreads;
    if (MN) { k = idx / (R / 8); mn = idx % (R / 8) * 8; }
    else    { mn = idx / 8; k = idx % 8 * 8; }
  }
  // Plain loads: a programmatic dependent starts before its input is complete, so no read may count as constant.
  __device__ __forceinline__ void load(const float* src, long long ld, int mn0, int mn_end, int k0, int k_end, int vec) {
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      int mn, k;
      place(i, mn, k);
      mn += mn0; k += k0;
      const float* g = src + (MN ? (long long)k * ld + mn : (long long)mn * ld + k);
      const int room = MN ? (k < k_end ? mn_end - mn : 0) : (mn < mn_end ? k_end - k : 0);   // elements there are
      if (vec && room >= 8) {
        *reinterpret_cast<float4*>(&v[i][0]) = *reinterpret_cast<const float4*>(g);
        *reinterpret_cast<float4*>(&v[i][4]) = *reinterpret_cast<const float4*>(g + 4);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = j < room ? g[j] : 0.0f;
      }
    }
  }
  __device__ __forceinline__ void split(uint8_t* parts) const {
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      int mn, k;
      place(i, mn, k);
      const int off = MN ? (mn >> 6) * (kTcBK * 128) + k * 128 + ((((mn >> 3) & 7) ^ (k & 7)) << 4)
                         : mn * 128 + (((k >> 3) ^ (mn & 7)) << 4);
      uint32_t p[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float a = v[i][2 * j], b = v[i][2 * j + 1];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          const uint32_t u = pack_bf16x2(a, b);
          p[s][j] = u;
          a -= __uint_as_float(u << 16);
          b -= __uint_as_float(u & 0xffff0000u);
        }
      }
#pragma unroll
      for (int s = 0; s < 3; ++s)
        *reinterpret_cast<uint4*>(parts + s * (R * 128) + off) = make_uint4(p[s][0], p[s][1], p[s][2], p[s][3]);
    }
  }
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// One output as one run of multiply-adds over all of K.
template <bool AMN, bool BMN>
__device__ __noinline__ float run_of_fma(const float* A, const float* B, long long lda, long long ldb, int K, int row, int col) {
  const float* a = A + (AMN ? row : row * lda);
  const float* b = B + (BMN ? col : col * ldb);
  float t = 0.0f;
  for (int k = 0; k < K; ++k) t = fmaf(AMN ? a[k * lda] : a[k], BMN ? b[k * ldb] : b[k], t);
  return t;
}
// Whether a sum may stand: zero, or between 2^-100 and the largest finite value.
__device__ __forceinline__ bool stands(float x) {
  const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
  return u == 0 || u - 0x0d800000u < 0x7f800000u - 0x0d800000u;
}

template <int BN, bool AMN, bool BMN>
__global__ void __launch_bounds__(kTcThreads + 32, 1)
gemm_f32_tc_kernel(const GemmF32Params p) {
  using L = TcF32Smem<BN>;
  constexpr int COLS = BN / 4;                       // columns of a thread: four warps share a lane quarter of TMEM
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBarOff);     // [2]: a k-block's parts are in shared memory
  uint64_t* done = full + 2;                                           // [2]: its MMAs have completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full[s], kTcThreads / 32);
      mbar_init(&done[s], 1);
    }
    mbar_fence_init();
  }
  if (warp == kTcThreads / 32) tmem_alloc<2 * BN>(tmem_slot);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  // As a programmatic dependent an x W^T product requests its first weights, which no kernel of a chain writes, before the wait.
  constexpr bool kAhead = !AMN && !BMN;
  if (!kAhead || warp == kTcThreads / 32) {
    pdl_wait();              // (programmatic dependent launch: no-ops in an ordinary launch)
    pdl_launch_dependents();
  }

  const int m0 = blockIdx.y * kTcBM, n0 = blockIdx.x * BN;
  const int k_begin = blockIdx.z * p.k_per_split;
  const int k_end = min(p.K, k_begin + p.k_per_split);
  const int blocks = (k_end - k_begin + kTcBK - 1) / kTcBK;
  float* out = reinterpret_cast<float*>(smem);       // [kTcBM][kOutLd]: this part's sums, once the stages are free

  if (warp == kTcThreads / 32) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(kTcBM, BN, AMN, BMN);
      int issued = 0;
      for (int i = 0; i < blocks; ++i) {
        // (accumulator i & 1 is free too: the warps arrive here after they have added block i - 2)
        if (!mbar_wait(&full[i & 1], (i >> 1) & 1, abort_flag, kWaitFullTimeout)) break;
        tc_fence_after_sync();
        const uint32_t a0 = smem_u32(smem + (i & 1) * L::kStage), b0 = a0 + 3 * L::kAPart, d = tmem + (i & 1) * BN;
        const int steps = (min(kTcBK, k_end - k_begin - i * kTcBK) + 15) / 16;
        // h l, l h, m m, h m, m h, h h
        constexpr int kA[6] = {0, 2, 1, 0, 1, 0}, kB[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
        for (int c = 0; c < 6; ++c)
#pragma unroll
          for (int kk = 0; kk < kTcBK / 16; ++kk) {
            const uint32_t a = a0 + kA[c] * L::kAPart, b = b0 + kB[c] * L::kBPart;
            if (kk < steps)
              umma_bf16(d, AMN ? make_smem_desc(a + kk * 2048, kTcBK * 128, 1024) : make_smem_desc(a + kk * 32, 16, 1024),
                        BMN ? make_smem_desc(b + kk * 2048, kTcBK * 128, 1024) : make_smem_desc(b + kk * 32, 16, 1024), idesc,
                        (c | kk) != 0);
          }
        umma_commit(&done[i & 1]);
        issued = i + 1;
      }
      if (*abort_flag && issued > 0) {
        const uint64_t t0 = global_timer_ns();
        while (!mbar_try_wait(&done[(issued - 1) & 1], ((issued - 1) >> 1) & 1) && global_timer_ns() - t0 < kWaitLimitNs / 4) {}
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ fetch, split, add
    const uint32_t t_row = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * COLS;
    float acc[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
    SplitTile<kTcBM, AMN> ta;
    SplitTile<BN, BMN> tb;
    // Adds the sums of k-block `i` once its MMAs have completed.
    auto collect = [&](int i) -> bool {
      if (!__all_sync(0xffffffffu, mbar_wait(&done[i & 1], (i >> 1) & 1, abort_flag, kWaitTmemFullTimeout))) return false;
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < COLS; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(t_row + (i & 1) * BN + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
      }
      tc_fence_before_sync();
      return true;
    };

    tb.load(p.B, p.ldb, n0, p.N, k_begin, k_end, p.vec_b);
    if (kAhead) {
      pdl_wait();
      pdl_launch_dependents();
    }
    ta.load(p.A, p.lda, m0, p.M, k_begin, k_end, p.vec_a);
    bool ok = true;
    for (int i = 0; i < blocks && ok; ++i) {
      // (stage i & 1 is free: `collect` of block i - 2 has waited for the MMAs that read it)
      uint8_t* stage = smem + (i & 1) * L::kStage;
      const int k1 = k_begin + (i + 1) * kTcBK;
      ta.split(stage);
      if (i + 1 < blocks) ta.load(p.A, p.lda, m0, p.M, k1, k_end, p.vec_a);
      tb.split(stage + 3 * L::kAPart);
      if (i + 1 < blocks) tb.load(p.B, p.ldb, n0, p.N, k1, k_end, p.vec_b);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[i & 1]);
      if (i > 0) ok = collect(i - 1);
    }
    if (ok && blocks > 0) ok = collect(blocks - 1);
    // (every MMA has completed: the last block's are the last; in a CTA that gave up the sums are worthless anyhow)
    float* row = out + ((warp & 3) * 32 + lane) * L::kOutLd + (warp >> 2) * COLS;
#pragma unroll
    for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4*>(row + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
  }
  tc_fence_before_sync();
  if (p.splits > 1) cluster_sync_all();
  else __syncthreads();
  if (warp == kTcThreads / 32) {
    tc_fence_after_sync();
    tmem_dealloc<2 * BN>(tmem);
  }

  constexpr int VECS = BN / 4;                       // 16-byte groups of a row
  const int rows = min(kTcBM, p.M - m0);
  for (int e = blockIdx.z * kTcThreads + threadIdx.x; e < rows * VECS && warp < kTcThreads / 32; e += p.splits * kTcThreads) {
    const int r = e / VECS, c = e % VECS * 4;
    const int row = m0 + r, col = n0 + c;
    if (col >= p.N) continue;
    const float* at = out + r * L::kOutLd + c;
    float4 v;
    if (p.splits > 1) {
      float4 q[kTcMaxSplits];                        // all requested before the first is used
#pragma unroll
      for (int s = 0; s < kTcMaxSplits; ++s)
        if (s < p.splits) q[s] = ld_cluster_v4(map_to_cta(at, s));
      v = q[0];
#pragma unroll
      for (int s = 1; s < kTcMaxSplits; ++s)
        if (s < p.splits) { v.x += q[s].x; v.y += q[s].y; v.z += q[s].z; v.w += q[s].w; }
    } else {
      v = *reinterpret_cast<const float4*>(at);
    }
    if (!(stands(v.x) & stands(v.y) & stands(v.z) & stands(v.w))) {
      v.x = run_of_fma<AMN, BMN>(p.A, p.B, p.lda, p.ldb, p.K, row, col);
      if (col + 1 < p.N) v.y = run_of_fma<AMN, BMN>(p.A, p.B, p.lda, p.ldb, p.K, row, col + 1);
      if (col + 2 < p.N) v.z = run_of_fma<AMN, BMN>(p.A, p.B, p.lda, p.ldb, p.K, row, col + 2);
      if (col + 3 < p.N) v.w = run_of_fma<AMN, BMN>(p.A, p.B, p.lda, p.ldb, p.K, row, col + 3);
    }
    if (p.vec_c && col + 3 < p.N) {
      epilogue_f32x4(p, row, col, v);
    } else {
      const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col + j < p.N) epilogue_f32(p, row, col + j, o[j]);
    }
  }
  if (p.splits > 1) cluster_sync_all();              // no CTA leaves while another reads its partial tile
}

template <int BN, bool AMN, bool BMN>
static cudaError_t launch_one(const GemmF32Params& p, cudaStream_t st) {
  using L = TcF32Smem<BN>;
  auto kern = gemm_f32_tc_kernel<BN, AMN, BMN>;
  static SmemLimit limit;
  const cudaError_t e = limit.raise(reinterpret_cast<const void*>(kern), L::kTotal);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = p.splits;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + BN - 1) / BN, (p.M + kTcBM - 1) / kTcBM, p.splits);
  cfg.blockDim = dim3(kTcThreads + 32);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = pdl_flag() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}
template <int BN>
static cudaError_t launch_bn(const GemmF32Params& p, bool amn, bool bmn, cudaStream_t st) {
  return amn ? (bmn ? launch_one<BN, true, true>(p, st) : launch_one<BN, true, false>(p, st))
             : (bmn ? launch_one<BN, false, true>(p, st) : launch_one<BN, false, false>(p, st));
}
// Clusters of `splits` CTAs that can be resident at once: they do not cross the GPC boundaries, so fewer CTAs than SMs.
template <int BN>
static int resident_clusters(int splits) {
  using L = TcF32Smem<BN>;
  static std::atomic<int> known[16][kTcMaxSplits + 1];   // one more than the number; 0: not asked for yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 16) return 0;
  int n = known[dev][splits].load(std::memory_order_relaxed) - 1;
  if (n < 0) {
    auto kern = gemm_f32_tc_kernel<BN, false, false>;
    static SmemLimit limit;
    if (limit.raise(reinterpret_cast<const void*>(kern), L::kTotal) != cudaSuccess) return 0;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = splits;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count(), 1, splits);
    cfg.blockDim = dim3(kTcThreads + 32);
    cfg.dynamicSmemBytes = L::kTotal;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known[dev][splits].store(n + 1, std::memory_order_relaxed);
  }
  return n;
}

// Microseconds that the best tile and split are expected to take: a wave of CTAs costs 6 us (launch, first loads, the last block's
// sums, the parts' meeting) and each of its k-blocks 1.68 us at BN = 64, 2.03 us at BN = 128.  Measured (B200), x W^T, each with the
// split this picks: 509 x 768 x 768 13.2 us (multiply-adds 21.9), 509 x 2304 x 768 20.1 (48.7), 509 x 3072 x 768 31.5 (60.0), 509 x 768
// x 3072 31.7 (65.5), 1024 x 256 x 1024 13.3 (22.7), 1024 x 256 x 256 7.7 (10.4), 256 x 256 x 1024 9.8 (11.9), 2048^3 144 (352).
double f32_tc_plan(int M, int N, int K, int* bn, int* splits) {
  double best = 1e300;
  const int kb = (K + kTcBK - 1) / kTcBK;
  for (int w = 64; w <= 128; w += 64) {
    const long long tiles = (long long)((M + kTcBM - 1) / kTcBM) * ((N + w - 1) / w);
    for (int s = 1; s <= kTcMaxSplits && s <= kb; ++s) {
      const int per = (kb + s - 1) / s;
      if ((kb + per - 1) / per != s) continue;               // some part would be empty
      const int n = w == 64 ? resident_clusters<64>(s) : resident_clusters<128>(s);
      if (n <= 0) continue;
      const double us = (double)((tiles + n - 1) / n) * (6.0 + per * (w == 64 ? 1.68 : 2.03));
      if (us < best) { best = us; *bn = w; *splits = s; }
    }
  }
  return best;
}

cudaError_t launch_f32_tc(const GemmF32Params& p, int bn, bool amn, bool bmn, cudaStream_t st) {
  return bn == 64 ? launch_bn<64>(p, amn, bmn, st) : launch_bn<128>(p, amn, bmn, st);
}

}  // namespace dptb
