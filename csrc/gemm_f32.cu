// fp32 GEMM, every operand layout, with a fused fp32 epilogue:
//
//   C[M,N] = epilogue( op(A)[M,K] * op(B)[K,N] ),   epilogue: *alpha, +bias, aux_out <- value, act, *act'(aux_in),
//                                                             +residual, (+C)
//
// (reference: lib/native/src/kernels/matmul.cuh:27-63, one 32x32 shared-memory tile and a separate kernel for each step of the
// epilogue.)
//
// The kernels of this file are multiply-adds: every one an IEEE fma into one accumulator per output and split of K, the splits
// added in order.  Two by the number of rows:
//   M <= 8   x W^T only: one pass over W at memory speed, a warp (or four) per pair of weight rows, no tiles.
//   else     tiles of 128x128 (8x8 outputs per thread), 64x64 (8x4) or 32x64 (4x4), double-buffered through shared
//            memory; operands are kept k-major there, swizzled so that both a K-contiguous operand (transposed on the
//            way in) and an M/N-contiguous one are stored and read without bank conflicts.
// What bounds the tiles is the issue of multiply-adds: fma.rn.f32x2 does two per instruction, which leaves issue slots
// for the shared-memory loads beside them.  From 256 terms on, where a tile's multiply-adds outweigh its launch, the tensor cores
// take over (gemm_f32_tc.cu).
#include <cuda_bf16.h>

#include "common/gemm_args.h"
#include "common/host.h"
#include "common/ptx.cuh"
#include "common/reduce.cuh"
#include "gemm_f32.cuh"

namespace dptb {

constexpr int kF32BK = 16;
// Below this many terms every output is one run of fma over K whatever the number of rows, so a row's bits do not depend on which
// others are computed with it (a decoder of width below 256 gives the same bits for some rows as for all).  From here on the
// streaming kernel, the tiles and each split add in an order of their own.  The line is where that property is given up for speed,
// not where the speed begins.  Measured (B200): 1 x 768 x K, K = 64 / 128 / 256: tiles 3.8 / 5.7 / 10 us, streaming 2.3 / 2.3 / 2.4 us;
// 8 rows 4.2 / 6.1 / 10 and 2.9 / 3.0 / 3.1 us; 256 x 256 x K, K = 128 / 192 / 256: one run 6.2 / 8.1 / 10.1 us, split 6.7 / 7.0 / 7.4 us.
constexpr int kOneRunK = 256;

// Position of element `mn` of k-row `k` in a shared tile of `R` elements per k-row: bits 3-4 are flipped by k / 4.  The
// four k-groups that a warp stores at once from a K-contiguous operand then fall on different banks, and 4-element
// groups stay whole for the reads.
__device__ __forceinline__ int f32_swz(int k, int mn) { return mn ^ (((k >> 2) & 3) << 3); }

// One operand tile [R x kF32BK] through registers.  MN: the operand's M / N axis is contiguous, else its K axis.
template <int R, int THREADS, bool MN>
struct F32Tile {
  static constexpr int kVecs = R * kF32BK / 4 / THREADS;
  static_assert(R * kF32BK / 4 % THREADS == 0, "whole 16-byte groups per thread");
  float4 v[kVecs];

  // Plain loads: a programmatic dependent starts before its input is complete, so no read may count as constant.
  __device__ __forceinline__ void load(const float* src, long long ld, int mn0, int mn_end, int k0, int k_end,
                                       int vec) {
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const int idx = threadIdx.x + i * THREADS;
      float e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (MN) {
        const int k = k0 + idx / (R / 4), mn = mn0 + idx % (R / 4) * 4;
        const float* g = src + (long long)k * ld + mn;
        if (k < k_end) {
          if (vec && mn + 3 < mn_end) {
            v[i] = *reinterpret_cast<const float4*>(g);
            continue;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (mn + j < mn_end) e[j] = g[j];
        }
      } else {
        const int mn = mn0 + idx / (kF32BK / 4), k = k0 + idx % (kF32BK / 4) * 4;
        const float* g = src + (long long)mn * ld + k;
        if (mn < mn_end) {
          if (vec && k + 3 < k_end) {
            v[i] = *reinterpret_cast<const float4*>(g);
            continue;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (k + j < k_end) e[j] = g[j];
        }
      }
      v[i] = make_float4(e[0], e[1], e[2], e[3]);
    }
  }
  __device__ __forceinline__ void store(float* s) const {
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const int idx = threadIdx.x + i * THREADS;
      if (MN) {
        const int k = idx / (R / 4), mn = idx % (R / 4) * 4;
        *reinterpret_cast<float4*>(s + k * R + f32_swz(k, mn)) = v[i];
      } else {
        const int mn = idx / (kF32BK / 4), k = idx % (kF32BK / 4) * 4;
        const int at = f32_swz(k, mn);
        s[k * R + at] = v[i].x;
        s[(k + 1) * R + at] = v[i].y;
        s[(k + 2) * R + at] = v[i].z;
        s[(k + 3) * R + at] = v[i].w;
      }
    }
  }
};

template <int BM, int BN, int TM, int TN, bool AMN, bool BMN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 512 / ((BM / TM) * (BN / TN)))
gemm_f32_kernel(const GemmF32Params p) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  constexpr int GM = TM / 4, GN = TN / 4;            // groups of four rows / columns, BM / GM and BN / GN apart
  constexpr int TX = BN / TN;                        // threads along N
  constexpr int WX = 8;                              // a warp covers 4 x 8 threads
  __shared__ __align__(16) float As[2][kF32BK * BM];
  __shared__ __align__(16) float Bs[2][kF32BK * BN];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = (warp % (TX / WX)) * WX + (lane & 7), ty = (warp / (TX / WX)) * 4 + (lane >> 3);
  pdl_wait();                // (programmatic dependent launch: no-ops in an ordinary launch)
  pdl_launch_dependents();
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int k_begin = blockIdx.z * p.k_per_split;
  const int k_end = min(p.K, k_begin + p.k_per_split);

  f32x2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  F32Tile<BM, THREADS, AMN> ta;
  F32Tile<BN, THREADS, BMN> tb;
  if (k_begin < k_end) {
    ta.load(p.A, p.lda, m0, p.M, k_begin, k_end, p.vec_a);
    tb.load(p.B, p.ldb, n0, p.N, k_begin, k_end, p.vec_b);
    ta.store(As[0]);
    tb.store(Bs[0]);
  }
  __syncthreads();
  int buf = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += kF32BK) {
    const bool more = k0 + kF32BK < k_end;
    if (more) {
      ta.load(p.A, p.lda, m0, p.M, k0 + kF32BK, k_end, p.vec_a);
      tb.load(p.B, p.ldb, n0, p.N, k0 + kF32BK, k_end, p.vec_b);
    }
    const float* as = As[buf];
    const float* bs = Bs[buf];
#pragma unroll      // (all 16 steps: 2048^3 353 us, 401 us by 8 and 431 us by 4)
    for (int k = 0; k < kF32BK; ++k) {
      float a[TM];
      f32x2 b[TN / 2];
#pragma unroll
      for (int g = 0; g < GM; ++g)
        *reinterpret_cast<float4*>(&a[g * 4]) = *reinterpret_cast<const float4*>(as + k * BM + f32_swz(k, g * (BM / GM) + ty * 4));
#pragma unroll
      for (int g = 0; g < GN; ++g)
        *reinterpret_cast<ulonglong2*>(&b[g * 2]) =
            *reinterpret_cast<const ulonglong2*>(bs + k * BN + f32_swz(k, g * (BN / GN) + tx * 4));
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const f32x2 ai = f2_splat(a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = f2_fma(ai, b[j], acc[i][j]);
      }
    }
    if (more) {
      ta.store(As[buf ^ 1]);
      tb.store(Bs[buf ^ 1]);
    }
    __syncthreads();
    buf ^= 1;
  }

  float4 out[TM][GN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int g = 0; g < GN; ++g) {
      f2_unpack(acc[i][g * 2], out[i][g].x, out[i][g].y);
      f2_unpack(acc[i][g * 2 + 1], out[i][g].z, out[i][g].w);
    }

  if (p.splits > 1) {
    // Partial tiles in thread order; the last CTA of a tile adds them in split order (the result does not depend on
    // which one that is) and runs the epilogue.
    const int tile = blockIdx.y * gridDim.x + blockIdx.x;
    float4* ws = reinterpret_cast<float4*>(p.ws) + (long long)tile * p.splits * (BM * BN / 4);
    float4* mine = ws + (long long)blockIdx.z * (BM * BN / 4) + threadIdx.x;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int g = 0; g < GN; ++g) mine[(i * GN + g) * THREADS] = out[i][g];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const int seen = atomicAdd(p.counters + tile, 1);
      s_last = seen == p.splits - 1;
      if (s_last) p.counters[tile] = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const float4* part = ws + threadIdx.x;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int g = 0; g < GN; ++g) out[i][g] = __ldcg(part + (i * GN + g) * THREADS);
    for (int s = 1; s < p.splits; ++s) {
      part += BM * BN / 4;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int g = 0; g < GN; ++g) {
          const float4 q = __ldcg(part + (i * GN + g) * THREADS);
          out[i][g].x += q.x; out[i][g].y += q.y; out[i][g].z += q.z; out[i][g].w += q.w;
        }
    }
  }

#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = m0 + (i / 4) * (BM / GM) + ty * 4 + (i & 3);
    if (row >= p.M) continue;
#pragma unroll
    for (int g = 0; g < GN; ++g) {
      const int col = n0 + g * (BN / GN) + tx * 4;
      if (p.vec_c && col + 3 < p.N) {
        epilogue_f32x4(p, row, col, out[i][g]);
      } else {
        const float v[4] = {out[i][g].x, out[i][g].y, out[i][g].z, out[i][g].w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < p.N) epilogue_f32(p, row, col + j, v[j]);
      }
    }
  }
}

// x W^T for up to MR <= 8 rows of x: WPR warps share kRowsPerWarp rows of W, each lane 16 bytes of every row at a time.
// Bound by reading W once; x comes from L1.  The lanes' sums meet in a fixed order.
constexpr int kVecThreads = 256;
template <int MR, int WPR, int ROWS>
__global__ void __launch_bounds__(kVecThreads)
gemv_f32_kernel(const GemmF32Params p) {
  constexpr int GROUPS = kVecThreads / 32 / WPR;
  __shared__ float part[kVecThreads / 32][ROWS * MR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp / WPR, sub = warp % WPR;
  const int n0 = (blockIdx.x * GROUPS + group) * ROWS;
  // The weights do not depend on the kernel before this one: as a programmatic dependent the first of them are under way
  // while that one finishes.
  constexpr int PRE = MR <= 4 ? 4 : 1, STEP = WPR * 128;
  const float* w[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) w[r] = p.B + (long long)min(n0 + r, p.N - 1) * p.ldb;
  const int kv = (p.vec_a && p.vec_b) ? p.K / 4 * 4 : 0, k_first = (sub * 32 + lane) * 4;
  float4 pre[PRE][ROWS];
#pragma unroll
  for (int u = 0; u < PRE; ++u)
    if (k_first + u * STEP < kv) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r) pre[u][r] = __ldg(reinterpret_cast<const float4*>(w[r] + k_first + u * STEP));
    }
  pdl_wait();
  pdl_launch_dependents();
  float acc[ROWS][MR];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[r][m] = 0.0f;
  if (n0 < p.N) {
    const float* x[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) x[m] = p.A + (long long)min(m, p.M - 1) * p.lda;
    auto add = [&](const float4 (&wv)[ROWS], int k) {
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const float4 xv = *reinterpret_cast<const float4*>(x[m] + k);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          acc[r][m] = fmaf(wv[r].x, xv.x, acc[r][m]);
          acc[r][m] = fmaf(wv[r].y, xv.y, acc[r][m]);
          acc[r][m] = fmaf(wv[r].z, xv.z, acc[r][m]);
          acc[r][m] = fmaf(wv[r].w, xv.w, acc[r][m]);
        }
      }
    };
#pragma unroll
    for (int u = 0; u < PRE; ++u)
      if (k_first + u * STEP < kv) add(pre[u], k_first + u * STEP);
#pragma unroll 4
    for (int k = k_first + PRE * STEP; k < kv; k += STEP) {
      float4 wv[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) wv[r] = __ldg(reinterpret_cast<const float4*>(w[r] + k));
      add(wv, k);
    }
    for (int k = kv + sub * 32 + lane; k < p.K; k += WPR * 32) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float wk = __ldg(w[r] + k);
#pragma unroll
        for (int m = 0; m < MR; ++m) acc[r][m] = fmaf(wk, x[m][k], acc[r][m]);
      }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const float t = warp_sum(acc[r][m]);
        if (lane == 0) part[warp][r * MR + m] = t;
      }
  }
  __syncthreads();
  const int e = threadIdx.x;                       // one output per thread
  if (e < GROUPS * ROWS * MR) {
    const int g = e / (ROWS * MR), i = e % (ROWS * MR);
    const int n = (blockIdx.x * GROUPS + g) * ROWS + i / MR, m = i % MR;
    if (n < p.N && m < p.M) {
      float t = part[g * WPR][i];
#pragma unroll
      for (int s = 1; s < WPR; ++s) t += part[g * WPR + s][i];
      epilogue_f32(p, m, n, t);
    }
  }
}

// Values before a GELU -> its derivative there, in place.
__global__ void __launch_bounds__(256)
gelu_slope_f32_kernel(float* __restrict__ x, long long ld, int M, int N) {
  const long long n = (long long)M * N, step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    float* p = x + i / N * ld + i % N;
    *p = act_grad_f32(12, *p);
  }
}

template <int MR, int ROWS>
static cudaError_t launch_gemv(const GemmF32Params& p, cudaStream_t st) {
  // One warp per group of rows when that fills the SMs with at least two CTAs each, else four.
  const int groups = (p.N + ROWS - 1) / ROWS;
  return groups >= sm_count() * 16 ? launch_k(gemv_f32_kernel<MR, 1, ROWS>, dim3((groups + 7) / 8), dim3(kVecThreads), 0, st, p)
                                   : launch_k(gemv_f32_kernel<MR, 4, ROWS>, dim3((groups + 1) / 2), dim3(kVecThreads), 0, st, p);
}

template <int BM, int BN, int TM, int TN>
static cudaError_t launch_tiles(const GemmF32Params& p, bool amn, bool bmn, cudaStream_t st) {
  const dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, p.splits);
  constexpr int T = (BM / TM) * (BN / TN);
  const auto kern = amn ? (bmn ? gemm_f32_kernel<BM, BN, TM, TN, true, true> : gemm_f32_kernel<BM, BN, TM, TN, true, false>)
                        : (bmn ? gemm_f32_kernel<BM, BN, TM, TN, false, true> : gemm_f32_kernel<BM, BN, TM, TN, false, false>);
  return launch_k(kern, grid, dim3(T), 0, st, p);
}

}  // namespace dptb

using namespace dptb;

static int product_f32(const DptbGemmArgs* a, cudaStream_t st) {
  GemmF32Params p;
  p.A = static_cast<const float*>(a->A);
  p.B = static_cast<const float*>(a->B);
  p.C = static_cast<float*>(a->C);
  p.bias = a->bias; p.bias_f32 = a->bias_f32;
  p.residual = static_cast<const float*>(a->residual); p.ldr = a->ldr;
  p.aux_out = static_cast<float*>(a->aux_out); p.ld_aux_out = a->ld_aux_out;
  p.aux_in = static_cast<const float*>(a->aux_in); p.ld_aux_in = a->ld_aux_in;
  p.lda = a->lda; p.ldb = a->ldb; p.ldc = a->ldc;
  p.M = a->M; p.N = a->N; p.K = a->K;
  p.accumulate = a->accumulate; p.act = a->act; p.alpha = a->alpha;
  auto vec = [](const void* q, long long ld) { return !q || ((reinterpret_cast<uintptr_t>(q) & 15) == 0 && ld % 4 == 0); };
  p.vec_a = vec(p.A, p.lda);
  p.vec_b = vec(p.B, p.ldb);
  p.vec_c = vec(p.C, p.ldc) && vec(p.residual, p.ldr) && vec(p.aux_out, p.ld_aux_out) && vec(p.aux_in, p.ld_aux_in);
  p.ws = static_cast<float*>(a->ws);
  p.counters = a->counters;
  p.splits = 1;
  p.k_per_split = (a->K + kF32BK - 1) / kF32BK * kF32BK;
  const bool amn = a->trans_a != 0, bmn = a->trans_b == 0;

  if (a->M <= 8 && a->K >= kOneRunK && !amn && !bmn && a->bn == 0 && a->splits <= 1) {
    return counted(1, (int)(a->M == 1 ? launch_gemv<1, 2>(p, st) : a->M == 2 ? launch_gemv<2, 2>(p, st)
                          : a->M <= 4 ? launch_gemv<4, 2>(p, st) : launch_gemv<8, 2>(p, st)));
  }

  // Tile and split of K by a small model of an SM: the CTAs that land on the busiest one share its multiply-add
  // units, which 16 resident warps keep busy; `rate` is the share of their peak that the tile's inner loop reaches, between what
  // 4096 x 4096 x K gives in one run at K = 2048 (B200: 51.4, 46.2 and 33.8 of 74.5 TFLOP/s: 0.69, 0.62, 0.45) and at K = 256 (0.63,
  // 0.58, 0.43).
  struct Tile { int bm, bn, warps; double rate; };
  static const Tile kTiles[3] = {{128, 128, 8, 0.70}, {64, 64, 4, 0.57}, {32, 64, 4, 0.42}};
  const int sms = sm_count();
  int best = 1, best_sp = 1;
  double best_cost = 1e300;
  for (int t = 0; t < 3; ++t) {
    if ((a->bn == 128 || a->bn == 64 || a->bn == 32) && kTiles[t].bm != a->bn) continue;
    const long long tiles = (long long)((a->M + kTiles[t].bm - 1) / kTiles[t].bm) * ((a->N + kTiles[t].bn - 1) / kTiles[t].bn);
    for (int sp = 1; sp <= 16; ++sp) {
      if (a->splits >= 1 && sp != a->splits) continue;
      if (sp > 1 && (!a->ws || !a->counters || tiles > a->num_counters ||
                     tiles * sp * kTiles[t].bm * kTiles[t].bn * 4 > a->ws_bytes || a->K / sp < 4 * kF32BK || (a->splits < 1 && a->K < kOneRunK)))
        break;
      const int k = ((a->K + sp - 1) / sp + kF32BK - 1) / kF32BK * kF32BK;
      const double area = (double)kTiles[t].bm * kTiles[t].bn;
      const double per_sm = (double)((tiles * sp + sms - 1) / sms);
      const double busy = per_sm * kTiles[t].warps / 16.0;
      const double clocks = per_sm * area * (k + 2 * kF32BK) / (128.0 * kTiles[t].rate * (busy < 1.0 ? 0.4 + 0.6 * busy : 1.0));
      // the fold: each split's tile leaves and comes back through L2
      const double fold = sp > 1 ? 2500.0 + area * 4.0 * sp / 64.0 : 0.0;
      if (clocks + fold < best_cost) { best_cost = clocks + fold; best = t; best_sp = sp; }
    }
  }
  // Tensor cores where they are expected to be faster (1.8 us: what the model above leaves out, launch and first loads).  Not below
  // kOneRunK, and not for forced tiles.  The few rows of a short step run as programmatic dependents, where set-up and first weights stand
  // beside the kernel ahead: 2 us less (an encoder of 6 layers, 23 rows of width 384: 314 us a pass with the multiply-add tiles, 296 so; 4
  // layers of width 768, 40 rows: 387 and 293; alone 23 x 384 x 384 takes 7.0 and 7.5 us).  By rows and not by the launch, so that both give
  // the same bits.
  if ((a->bn == 0 && a->splits < 1 && a->K >= kOneRunK) || a->bn == 1064 || a->bn == 1128) {
    int bn = a->bn - 1000, sp = a->splits < 1 ? 1 : a->splits;
    if (a->bn || f32_tc_plan(a->M, a->N, a->K, &bn, &sp) < best_cost / 1900.0 + (a->M <= 64 ? 3.8 : 1.8)) {
      const int kb = (a->K + kF32TcBK - 1) / kF32TcBK, per = kb > 0 ? (kb + sp - 1) / sp : 1;
      p.k_per_split = per * kF32TcBK;
      p.splits = kb > 0 ? (kb + per - 1) / per : 1;
      if (p.splits > 8 || (a->M + 127) / 128 > 65535) return kErrBadShape;
      return counted(1, (int)launch_f32_tc(p, bn, amn, bmn, st));
    }
  }
  p.k_per_split = ((a->K + best_sp - 1) / best_sp + kF32BK - 1) / kF32BK * kF32BK;
  p.splits = a->K > 0 ? (a->K + p.k_per_split - 1) / p.k_per_split : 1;   // every split non-empty
  if (p.k_per_split == 0) p.k_per_split = kF32BK;
  if ((a->M + kTiles[best].bm - 1) / kTiles[best].bm > 65535) return kErrBadShape;
  return counted(1, (int)(best == 0 ? launch_tiles<128, 128, 8, 8>(p, amn, bmn, st)
                        : best == 1 ? launch_tiles<64, 64, 8, 4>(p, amn, bmn, st) : launch_tiles<32, 64, 4, 4>(p, amn, bmn, st)));
}

// All operands, the output and the per-element buffers in fp32 (the bias may be bf16).  Any shape, any stride.
// GELU with its derivative (code 5) is GELU that saves its argument and a pass that turns it into the derivative: no model
// saves the derivative in fp32, and its arithmetic in the unrolled epilogues cost every other product about 1 us of
// instruction fetches (training step of 6 layers x 1024 rows x 256: 2.20 against 2.27 ms; encoder of 23 rows: 314 against 324 us).
int gemm_f32(const DptbGemmArgs* a, void* stream_v) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_v);
  if (a->act != 5) return product_f32(a, st);
  DptbGemmArgs g = *a;
  g.act = 2;
  const int rc = product_f32(&g, st);
  if (rc || !a->aux_out) return rc;
  const long long blocks = ((long long)a->M * a->N + 255) / 256, most = 8LL * sm_count();
  gelu_slope_f32_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, st>>>(static_cast<float*>(a->aux_out), a->ld_aux_out,
                                                                                  a->M, a->N);
  return counted(1, (int)cudaGetLastError());
}
