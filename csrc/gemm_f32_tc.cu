// fp32 GEMM on the tensor cores: operands split into three bf16 parts, products summed as closely as multiply-adds sum them.
//
// An fp32 value is exactly h + m + l with three bf16 parts of 8 significant bits each (rounded to nearest, so m and l may
// carry the other sign; the splitting of Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For
// Higher-Precision Computations", 2019).  Of the nine products of two such values six are formed, h h, h m, m h, m m, h l, l h; what is left
// out, m l + l m + l l, is below 2^-25 of the product, less than the rounding of one fp32 multiply.  Every bf16 product is exact; the
// accumulator is not: tcgen05 truncates where an fma rounds, so a long chain drifts towards zero.  Therefore the small
// products of a k-block go first (their truncations are 2^-8 of an ulp), h h last, in an accumulator for each half of the block, and after
// 64 terms both leave TMEM and are added in fp32 registers, rounded to nearest: two truncated steps, not K / 16, ever meet in one
// accumulator.  (With four, products of one sign, whose truncations add up, were further from fp64 than multiply-adds; 2048^3 took
// 156 us with them, 167 so.)
//
// A CTA computes a 128 x BN tile over one part of K.  Its 16 warps do everything: fetch the next k-block from global memory
// into registers, split the present one into shared memory (swizzled bf16 tiles in the operand's own orientation: K-major or
// MN-major descriptors, no transpose), one thread issues the 24 MMAs, and while they run all warps add the block before to
// their registers and split the next.  The parts of K are CTAs of one cluster: each leaves its partial tile in its own shared
// memory and every CTA of the cluster adds an equal share of the rows, in the order of the parts, and runs the epilogue on it.
// Deterministic, and no scratch in global memory.
//
// Not every value is the sum of three such parts: bits below 2^-133 have no bf16.  While it splits, a CTA marks the rows (of A and of
// B) with elements that are not zero and below 2^-110.  Outputs of marked rows, outputs that are not finite (infinity, NaN and what rounds
// to infinity in bf16 make NaN of their parts), and outputs that are not zero and below 2^-100, are computed again as multiply-adds:
// the cluster does its tile once more with them, the outputs concerned take those sums, and all others keep the bits that they have
// without such neighbours.
//
// Distance from fp64 (2-norm, relative; B200) against the multiply-add tiles with their splits: normal operands, 509 x 768 x 768 0.81e-7
// (2.1e-7), 509 x 768 x 3072 1.07e-7 (2.9e-7), 256 x 256 x 1024 0.85e-7 (1.6e-7); operands that are all positive, 509 x 768 x 768 0.60e-7
// (0.81e-7), 23 x 384 x 384 0.63e-7 (0.65e-7).
//
// What bounds it: shared memory.  A k-block at BN = 128 writes 96 KB of parts and its MMAs read 192 KB, 2300 clocks at 128 bytes
// each, against 1536 of the MMAs alone; fetching 64 KB ahead of the split only partly overlaps it (4500 clocks measured).  It is
// still 2.1 times the rate of the packed multiply-adds (2048^3: 352 -> 167 us).
#include "common/cluster_limit.h"
#include "gemm_f32.cuh"

namespace dptb {

constexpr int kTcBM = 128, kTcBK = kF32TcBK;
constexpr int kTcMaxSplits = 8;                      // CTAs of a cluster
constexpr int kTcThreads = 512;                      // 16 warps that fetch, split and add; one more issues the MMAs
constexpr int kRedoBK = 16;

template <int BN>
struct TcF32Smem {
  static constexpr int kAPart = kTcBM * 128, kBPart = BN * 128;     // one bf16 part of a k-block: 128 bytes a row
  static constexpr int kStage = 3 * (kAPart + kBPart);
  static constexpr int kOutLd = BN + 4;                            // floats; 16-byte rows, quarter-warps on different banks
  static constexpr int kBarOff = 2 * kStage;
  static constexpr int kAnyLostOff = kBarOff + 48, kRedoFlagOff = kBarOff + 52, kLostOff = kBarOff + 64;                    // a byte a row of A and of B: it has elements without three parts
  static constexpr int kTotal = kLostOff + kTcBM + BN + 1024;
  // The stages are used again: the partial tile, the same from multiply-adds, and their operands (kRedoBK terms, k-major).
  static constexpr int kRedoOff = kTcBM * kOutLd * 4, kRedoAOff = 2 * kRedoOff, kRedoBOff = kRedoAOff + kRedoBK * (kTcBM + 4) * 4;
  static_assert(kRedoBOff + kRedoBK * (BN + 4) * 4 <= 2 * kStage, "the partial tiles reuse the stages");
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
  // An element from 2^-110 on is the sum of its parts: its last bit is worth 2^-133 or more, the least that bf16 holds.  (The sign
  // shifted out, less one, so that zero is the largest.)
  static constexpr uint32_t kWhole = 2u * 0x08800000u - 1u;
  static __device__ __forceinline__ uint32_t doubled(float x) { return 2u * __float_as_uint(x) - 1u; }
  // `lost`: a byte for each of the R rows, set where an element is smaller and not zero.
  __device__ __forceinline__ void split(uint8_t* parts, uint8_t* lost, int* any_lost) const {
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      int mn, k;
      place(i, mn, k);
      const int off = MN ? (mn >> 6) * (kTcBK * 128) + k * 128 + ((((mn >> 3) & 7) ^ (k & 7)) << 4)
                         : mn * 128 + (((k >> 3) ^ (mn & 7)) << 4);
      uint32_t p[3][4], least = ~0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float a = v[i][2 * j], b = v[i][2 * j + 1];
        least = __vimin3_u32(least, doubled(a), doubled(b));
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          const uint32_t u = pack_bf16x2(a, b);
          p[s][j] = u;
          a -= __uint_as_float(u << 16);
          b -= __uint_as_float(u & 0xffff0000u);
        }
      }
      if (__builtin_expect(least < kWhole, 0)) {
        if (MN) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (doubled(v[i][j]) < kWhole) lost[mn + j] = 1;
        } else {
          lost[mn] = 1;
        }
        *any_lost = 1;
      }
#pragma unroll
      for (int s = 0; s < 3; ++s)
        *reinterpret_cast<uint4*>(parts + s * (R * 128) + off) = make_uint4(p[s][0], p[s][1], p[s][2], p[s][3]);
    }
  }
};

// The tile's sums over this CTA's part of K as multiply-adds, into `out` [kTcBM][kOutLd]: by the 16 warps, kRedoBK terms at a time, the
// next ones under way.  B200, a column of NaN in A: 509 x 768 x 768 57 us, 2048^3 901 us (15 and 167 without; multiply-add tiles alone 22 and 352).
template <int BN, bool AMN, bool BMN>
__device__ __noinline__ void multiply_add_tile(const GemmF32Params& p, uint8_t* smem, int m0, int n0, int k_begin, int k_end) {
  using L = TcF32Smem<BN>;
  constexpr int TX = BN / 4, ROWS = kTcBM * TX / kTcThreads;       // a thread: ROWS (8 or 4) rows of four columns
  constexpr int EA = kTcBM * kRedoBK / kTcThreads, EB = BN * kRedoBK / kTcThreads;
  float* out = reinterpret_cast<float*>(smem + L::kRedoOff);
  float* as = reinterpret_cast<float*>(smem + L::kRedoAOff);       // [kRedoBK][kTcBM + 4]
  float* bs = reinterpret_cast<float*>(smem + L::kRedoBOff);       // [kRedoBK][BN + 4]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;      // a warp: 4 x 8 threads
  const int tx = warp % (TX / 8) * 8 + (lane & 7), ty = warp / (TX / 8) * 4 + (lane >> 3);
  const float* const A = p.A;                                      // (read once: the barriers below make memory unknown)
  const float* const B = p.B;
  const long long lda = p.lda, ldb = p.ldb;
  const int M = p.M, N = p.N;
  float ra[EA], rb[EB];
  auto at = [](int i, int rows, bool mn_major, int& mn, int& k) {
    const int idx = threadIdx.x + i * kTcThreads;
    mn = mn_major ? idx % rows : idx / kRedoBK;
    k = mn_major ? idx / rows : idx % kRedoBK;
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < EA; ++i) {
      int mn, k;
      at(i, kTcBM, AMN, mn, k);
      mn += m0; k += k0;
      ra[i] = mn < M && k < k_end ? A[AMN ? (long long)k * lda + mn : (long long)mn * lda + k] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      int mn, k;
      at(i, BN, BMN, mn, k);
      mn += n0; k += k0;
      rb[i] = mn < N && k < k_end ? B[BMN ? (long long)k * ldb + mn : (long long)mn * ldb + k] : 0.0f;
    }
  };
  f32x2 acc[ROWS][2];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) acc[i][0] = acc[i][1] = 0ull;
  fetch(k_begin);
  for (int k0 = k_begin; k0 < k_end; k0 += kRedoBK) {
    __syncwarp();
    asm volatile("bar.sync 1, 512;" ::: "memory");
#pragma unroll
    for (int i = 0; i < EA; ++i) {
      int mn, k;
      at(i, kTcBM, AMN, mn, k);
      as[k * (kTcBM + 4) + mn] = ra[i];
    }
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      int mn, k;
      at(i, BN, BMN, mn, k);
      bs[k * (BN + 4) + mn] = rb[i];
    }
    __syncwarp();
    asm volatile("bar.sync 1, 512;" ::: "memory");
    if (k0 + kRedoBK < k_end) fetch(k0 + kRedoBK);
    const int terms = min(kRedoBK, k_end - k0);                    // (no term beyond K: 0 times infinity)
#pragma unroll 4
    for (int k = 0; k < terms; ++k) {
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bs + k * (BN + 4) + tx * 4);
      float a[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; i += 4)
        *reinterpret_cast<float4*>(&a[i]) = *reinterpret_cast<const float4*>(as + k * (kTcBM + 4) + ty * ROWS + i);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const f32x2 ai = f2_splat(a[i]);
        acc[i][0] = f2_fma(ai, b.x, acc[i][0]);
        acc[i][1] = f2_fma(ai, b.y, acc[i][1]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    float4 v;
    f2_unpack(acc[i][0], v.x, v.y);
    f2_unpack(acc[i][1], v.z, v.w);
    *reinterpret_cast<float4*>(out + (ty * ROWS + i) * L::kOutLd + tx * 4) = v;
  }
}
// Whether a sum may stand: zero, or between 2^-100 and the largest finite value.
__device__ __forceinline__ bool stands(float x) {
  const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
  return u == 0 || u - 0x0d800000u < 0x7f800000u - 0x0d800000u;
}

// Sum of the parts of K of four neighbouring outputs, in the order of the parts.
__device__ __forceinline__ float4 sum_of_parts(const float* at, int splits) {
  if (splits == 1) return *reinterpret_cast<const float4*>(at);
  float4 q[kTcMaxSplits];                        // all requested before the first is used
#pragma unroll
  for (int s = 0; s < kTcMaxSplits; ++s)
    if (s < splits) q[s] = ld_cluster_v4(map_to_cta(at, s));
  float4 v = q[0];
#pragma unroll
  for (int s = 1; s < kTcMaxSplits; ++s)
    if (s < splits) { v.x += q[s].x; v.y += q[s].y; v.z += q[s].z; v.w += q[s].w; }
  return v;
}
// This CTA's share of the tile's outputs; AGAIN: those that could not stand, as the sums of multiply-adds.
template <int BN, bool AGAIN>
__device__ __forceinline__ void finish_tile(const GemmF32Params& p, uint8_t* smem, int m0, int n0) {
  using L = TcF32Smem<BN>;
  constexpr int VECS = BN / 4;                       // 16-byte groups of a row
  const float* out = reinterpret_cast<const float*>(smem);
  const int rows = min(kTcBM, p.M - m0);
  for (int e = blockIdx.z * kTcThreads + threadIdx.x; e < rows * VECS; e += p.splits * kTcThreads) {
    const int r = e / VECS, c = e % VECS * 4;
    const int row = m0 + r, col = n0 + c;
    if (col >= p.N) continue;
    float4 v = sum_of_parts(out + r * L::kOutLd + c, p.splits);
    int todo = 15;
    if (AGAIN || !(stands(v.x) & stands(v.y) & stands(v.z) & stands(v.w))) {
      const int sick = (stands(v.x) ? 0 : 1) | (stands(v.y) ? 0 : 2) | (stands(v.z) ? 0 : 4) | (stands(v.w) ? 0 : 8);
      todo = AGAIN ? sick : 15 & ~sick;
      if (AGAIN) v = sum_of_parts(out + L::kRedoOff / 4 + r * L::kOutLd + c, p.splits);
      else
        for (int s = 0; s < p.splits; ++s) st_cluster_u32(map_to_cta(smem + L::kRedoFlagOff, s), 1);
    }
    if (!AGAIN && todo == 15 && p.vec_c && col + 3 < p.N) {
      epilogue_f32x4(p, row, col, v);
    } else {
      const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((todo >> j & 1) && col + j < p.N) epilogue_f32(p, row, col + j, o[j]);
    }
  }
}
template <int BN>
__device__ __noinline__ void finish_again(const GemmF32Params& p, uint8_t* smem, int m0, int n0) {
  finish_tile<BN, true>(p, smem, m0, n0);
}

template <int BN, bool AMN, bool BMN>
__global__ void __launch_bounds__(kTcThreads + 32, 1)
gemm_f32_tc_kernel(const __grid_constant__ GemmF32Params p) {
  using L = TcF32Smem<BN>;
  constexpr int COLS = BN / 4;                       // columns of a thread: four warps share a lane quarter of TMEM
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBarOff);     // [2]: a k-block's parts are in shared memory
  uint64_t* done = full + 2;                                           // [2]: its MMAs have completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* any_lost = reinterpret_cast<int*>(smem + L::kAnyLostOff);       // some element of this part has no three parts
  volatile int* redo = reinterpret_cast<volatile int*>(smem + L::kRedoFlagOff);   // some output of the cluster's tile is computed again
  uint8_t* lost = smem + L::kLostOff;                                  // [kTcBM] rows of A, [BN] of B
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < (kTcBM + BN) / 4) reinterpret_cast<uint32_t*>(lost)[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    *abort_flag = *any_lost = *redo = 0;
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full[s], kTcThreads / 32);
      mbar_init(&done[s], 1);
    }
    mbar_fence_init();
  }
  if (warp == kTcThreads / 32) tmem_alloc<4 * BN>(tmem_slot);
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
              umma_bf16(c == 5 && kk >= 2 ? d + 2 * BN : d, AMN ? make_smem_desc(a + kk * 2048, kTcBK * 128, 1024) : make_smem_desc(a + kk * 32, 16, 1024),
                        BMN ? make_smem_desc(b + kk * 2048, kTcBK * 128, 1024) : make_smem_desc(b + kk * 32, 16, 1024), idesc,
                        (c | kk) != 0 && !(c == 5 && kk == 2));
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
      const bool second = k_end - k_begin - i * kTcBK > 32;
#pragma unroll
      for (int c = 0; c < COLS; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(t_row + (i & 1) * BN + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
        if (second) {
          tmem_ld_32x16(t_row + (2 + (i & 1)) * BN + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
        }
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
      ta.split(stage, lost, any_lost);
      if (i + 1 < blocks) ta.load(p.A, p.lda, m0, p.M, k1, k_end, p.vec_a);
      tb.split(stage + 3 * L::kAPart, lost + kTcBM, any_lost);
      if (i + 1 < blocks) tb.load(p.B, p.ldb, n0, p.N, k1, k_end, p.vec_b);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[i & 1]);
      if (i > 0) ok = collect(i - 1);
    }
    if (ok && blocks > 0) ok = collect(blocks - 1);
    // (every MMA has completed: the last block's are the last; in a CTA that gave up the sums are worthless anyhow)
    __syncwarp();
    asm volatile("bar.sync 1, 512;" ::: "memory");   // (all marks are made)
    const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * COLS;
    if (__builtin_expect(*reinterpret_cast<volatile int*>(any_lost), 0)) {
      // what cannot stand becomes NaN, in whatever part of K it was seen
#pragma unroll
      for (int j = 0; j < COLS; ++j)
        if (lost[r] | lost[kTcBM + c0 + j]) acc[j] = __int_as_float(0x7fffffff);
    }
    float* row = out + r * L::kOutLd + c0;
#pragma unroll
    for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4*>(row + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
  }
  auto meet = [&] {
    if (p.splits > 1) cluster_sync_all();
    else __syncthreads();
  };
  tc_fence_before_sync();
  meet();
  if (warp == kTcThreads / 32) {
    tc_fence_after_sync();
    tmem_dealloc<4 * BN>(tmem);
  }

  if (warp < kTcThreads / 32) finish_tile<BN, false>(p, smem, m0, n0);
  meet();                                            // (no CTA leaves while another reads its partial tile)
  if (*redo) {
    if (warp < kTcThreads / 32) multiply_add_tile<BN, AMN, BMN>(p, smem, m0, n0, k_begin, k_end);
    meet();
    if (warp < kTcThreads / 32) finish_again<BN>(p, smem, m0, n0);
    meet();
  }
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
  static ClusterLimit limits[kTcMaxSplits + 1];
  static SmemLimit smem;
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
  return limits[splits].resident(reinterpret_cast<const void*>(gemm_f32_tc_kernel<BN, false, false>), smem, L::kTotal, cfg);
}

// Microseconds that the best tile and split are expected to take: a wave of CTAs costs 5.5 us at BN = 64, 8.0 us at BN = 128 (launch, first
// loads, the last block's sums, the parts' meeting) and each of its k-blocks 2.0 and 2.35 us.  Measured (B200), x W^T, each with the
// split this picks: 509 x 768 x 768 14.8 us (multiply-adds 21.8), 509 x 2304 x 768 22.8 (48.7), 509 x 3072 x 768 36.3 (60.1), 509 x 768
// x 3072 32.8 (65.8), 1024 x 256 x 1024 14.6 (22.7), 1024 x 256 x 256 8.3 (10.5), 256 x 256 x 1024 10.7 (11.9), 2048^3 167 (352).
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
      const double us = (double)((tiles + n - 1) / n) * (w == 64 ? 5.5 + 2.0 * per : 8.0 + 2.35 * per);
      if (us < best) { best = us; *bn = w; *splits = s; }
    }
  }
  return best;
}

cudaError_t launch_f32_tc(const GemmF32Params& p, int bn, bool amn, bool bmn, cudaStream_t st) {
  return bn == 64 ? launch_bn<64>(p, amn, bmn, st) : launch_bn<128>(p, amn, bmn, st);
}

}  // namespace dptb
