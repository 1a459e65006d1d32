// Attention in fp32, forward and backward (no tensor cores: every product and sum is an fp32 multiply-add).
//
// float32 is the default dtype of the models; these kernels replace a chain of launches per (batch, head): scale, mask, softmax and
// two products forward, twice that backward (reference: lib/core/tensor/attention.dart:39-53).  Operands are strided
// [batch, seq, head, hd] views (a fused projection output, a cache, separate tensors), head size up to 128, grouped queries.
//
//   attn_f32_fwd     CTA = 32 query rows of one (batch, head), walks tiles of 64 keys with a running maximum and sum.  Four CTAs
//                    fit an SM (51 KB each at heads of 64): what a launch of the composed chain cost in gaps, neighbours now hide.
//   attn_f32_decode  few query rows over a long history: a cluster of up to 8 CTAs shares the keys of one (batch, kv head), each
//                    streams its own tiles, and the partial results meet in distributed shared memory (no workspace, fixed order)
//   attn_f32_dq      CTA = 32 query rows, walks the keys: delta = rowsum(dO O), dQ
//   attn_f32_dkv     CTA = 64 keys of one (batch, kv head), walks the group's query rows: dK, dV.  Probabilities are recomputed in
//                    both kernels instead of meeting in fp32 atomics: results are the same from run to run.
//
// Bound: shared-memory reads and fp32 issue (a thread does 4 x 4 outputs: 8 16-byte reads for 64 multiply-adds, as 32 packed
// ones); at the sizes fp32 models run, the latency of a few tiles.  Measured as whole passes, chain per head -> these kernels:
// training step of 6 layers x 8 sequences x 8 heads x 128 tokens x 32: 64.6 -> 8.7 ms; GPT-2 124M, prompt of 509 tokens:
// 36.6 -> 12.4 ms, a token after it: 30.6 -> 11.9 ms (what was left there was the fp32 GEMM and host work: 2.1 and 0.45 ms since).
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "common/attn_args.h"
#include "common/host.h"
#include "common/ptx.cuh"

namespace dptb {
namespace cg = cooperative_groups;

struct F32View {          // element (b, s, h, d) at p[b * sb + s * ss + h * sh + d]
  float* p;
  long long sb, ss, sh;
};
struct AttnF32Params {
  F32View q, k, v, o, dout, dq, dk, dv;
  float* lse;             // [B, Hq, Sq]
  float* delta;           // [B, Hq, Sq]
  int B, Sq, Sk, Hq, Hkv, hd;
  int causal, q_offset;   // causal: key j is visible to query i when j <= i + q_offset
  float scale;
  int vec;                // every row starts on a 16-byte boundary and hd is a multiple of 4
  // Decoding only: the keys and values of the rows from `appended` on (Sk: none) are read from kn / vn (row 0 there) and written to
  // k / v, the caches.
  F32View kn, vn;
  int appended;
  int key_ctas;           // forward tiles: CTAs that share the keys of a row tile
};

constexpr int kFBM = 32, kFBN = 64, kFThreads = 128;
template <int HD> __host__ __device__ constexpr int f32_ld() { return HD + 4; }   // 4 floats of padding: 16-byte reads of 8 rows touch all banks once

// Rows [row0, row0 + ROWS) of head `h` into shared memory [ROWS][HD + 4]; zeros beyond `rows` and beyond hd.
template <int HD, int ROWS>
__device__ __forceinline__ void f32_load_tile(float* dst, const F32View& t, int b, int h, int row0, int rows, int hd, int vec) {
  const float* base = t.p + b * t.sb + h * t.sh;
  constexpr int C4 = HD / 4;
#pragma unroll 4
  for (int i = threadIdx.x; i < ROWS * C4; i += kFThreads) {
    const int r = i / C4, c = (i % C4) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row0 + r < rows) {
      const float* src = base + (row0 + r) * t.ss + c;
      if (vec) {
        if (c < hd) x = *reinterpret_cast<const float4*>(src);
      } else {
        if (c + 0 < hd) x.x = src[0];
        if (c + 1 < hd) x.y = src[1];
        if (c + 2 < hd) x.z = src[2];
        if (c + 3 < hd) x.w = src[3];
      }
    }
    *reinterpret_cast<float4*>(dst + r * f32_ld<HD>() + c) = x;
  }
}

// The same without waiting: copies under way when every row takes 16-byte accesses, else plain loads.
template <int HD, int ROWS>
__device__ __forceinline__ void f32_request_tile(float* dst, const F32View& t, int b, int h, int row0, int rows, int hd, int vec) {
  if (vec) {
    const float* base = t.p + b * t.sb + h * t.sh;
    constexpr int C4 = HD / 4;
#pragma unroll 4
    for (int i = threadIdx.x; i < ROWS * C4; i += kFThreads) {
      const int r = i / C4, c = (i % C4) * 4;
      const bool live = row0 + r < rows && c < hd;
      const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst + r * f32_ld<HD>() + c));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(live ? base + (row0 + r) * t.ss + c : base),
                   "r"(live ? 16 : 0) : "memory");
    }
  } else {
    f32_load_tile<HD, ROWS>(dst, t, b, h, row0, rows, hd, vec);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// acc[i][j] = A[ty * 4 + i] . B[tx + 16 j]
template <int HD>
__device__ __forceinline__ void f32_tile_dot(const float* A, const float* Bt, int ty, int tx, float (&acc)[4][4]) {
  constexpr int LD = f32_ld<HD>();
  f32x2 s[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0ull;
#pragma unroll 4
  for (int d = 0; d < HD; d += 4) {
    ulonglong2 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(A + (ty * 4 + i) * LD + d);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(Bt + (tx + 16 * j) * LD + d);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = f2_fma(a[i].y, b[j].y, f2_fma(a[i].x, b[j].x, s[i][j]));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      f2_unpack(s[i][j], lo, hi);
      acc[i][j] = lo + hi;
    }
}

// out[i][c] += sum over 64 keys of W[ty * 4 + i][key] * V[key][column c of this thread]; a thread owns HD / 16 columns in runs of
// up to 4 (tx * 4 + 64 m), so that a half warp reads whole rows.
template <int HD> struct F32Cols { static constexpr int N = HD / 16, RUN = N < 4 ? N : 4; };
template <int HD>
__device__ __forceinline__ int f32_col(int tx, int c) { return tx * F32Cols<HD>::RUN + (c / 4) * 64 + (c % 4); }
template <int HD>
__device__ __forceinline__ void f32_tile_acc(const float* W, const float* Vt, int ty, int tx, float (&out)[4][F32Cols<HD>::N]) {
  constexpr int LD = f32_ld<HD>(), N = F32Cols<HD>::N, RUN = F32Cols<HD>::RUN, LW = kFBN + 4;
#pragma unroll 2
  for (int k = 0; k < kFBN; k += 4) {
    float w[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(W + (ty * 4 + i) * LW + k);
      w[i][0] = x.x; w[i][1] = x.y; w[i][2] = x.z; w[i][3] = x.w;
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float v[N];
#pragma unroll
      for (int c = 0; c < N; c += RUN) {
        const float* src = Vt + (k + kk) * LD + f32_col<HD>(tx, c);
        if constexpr (RUN == 4) {
          const float4 x = *reinterpret_cast<const float4*>(src);
          v[c] = x.x; v[c + 1] = x.y; v[c + 2] = x.z; v[c + 3] = x.w;
        } else if constexpr (RUN == 2) {
          const float2 x = *reinterpret_cast<const float2*>(src);
          v[c] = x.x; v[c + 1] = x.y;
        } else {
          v[c] = *src;
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < N; ++c) out[i][c] = fmaf(w[i][kk], v[c], out[i][c]);
    }
  }
}

__device__ __forceinline__ float half_warp_max(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float half_warp_sum(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Key tiles that the rows [row0, row0 + 32) can see.
__host__ __device__ __forceinline__ int f32_key_tiles(const AttnF32Params& p, int row0) {
  int last = p.Sk - 1;
  const int end = row0 + kFBM < p.Sq ? row0 + kFBM : p.Sq;
  if (p.causal && end - 1 + p.q_offset < last) last = end - 1 + p.q_offset;
  return last < 0 ? 0 : last / kFBN + 1;
}

template <int HD, bool SHARED>
__global__ void __launch_bounds__(kFThreads)
attn_f32_fwd(const AttnF32Params p) {
  extern __shared__ float4 sm4[];
  constexpr int LD = f32_ld<HD>(), LW = kFBN + 4, N = F32Cols<HD>::N;
  float* Qs = reinterpret_cast<float*>(sm4);
  float* Ks = Qs + kFBM * LD;
  float* Vs = Ks + kFBN * LD;
  float* Ps = Vs + kFBN * LD;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  pdl_wait();                // (programmatic dependent launch: no-ops in an ordinary launch)
  pdl_launch_dependents();
  // The key tiles of the rows are dealt out to the CTAs of a cluster (one, two or four).  The units go by the length of their rows, all
  // heads of the longest first, so that the last ones to find an SM are the shortest (B200, causal, 12 heads of 64: 509 tokens 41.5 us
  // with the rows of each head together, 31.1 us so; 1024 tokens 96.5 and 80.3 us).
  const int nc = SHARED ? p.key_ctas : 1, rank = SHARED ? blockIdx.x % nc : 0, unit = blockIdx.x / nc;
  const int qx = unit / (p.B * p.Hq), bh = unit - qx * p.B * p.Hq;
  const int qt = p.causal ? (p.Sq + kFBM - 1) / kFBM - 1 - qx : qx;     // the longest rows of all heads start first
  const int b = bh / p.Hq, h = bh - b * p.Hq, hk = h / (p.Hq / p.Hkv), row0 = qt * kFBM;
  f32_load_tile<HD, kFBM>(Qs, p.q, b, h, row0, p.Sq, p.hd, p.vec);
  float m[4], l[4], o[4][N];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < N; ++c) o[i][c] = 0.f;
  }
  const int tiles = f32_key_tiles(p, row0);
  // K and V have a buffer each; a tile is requested as soon as its buffer has been read, so that it arrives under the other
  // product.  (The time of a key tile was that of fetching it: B200, causal, 12 heads of 64, 509 tokens: 51.6 us with
  // plain loads between two barriers, 42.3 us so; 256 tokens 22.3 and 16.3 us; 6 heads of 128, 509 tokens 73.5 and 49.0 us.)
  if (rank < tiles) {
    f32_request_tile<HD, kFBN>(Ks, p.k, b, hk, rank * kFBN, p.Sk, p.hd, p.vec);
    f32_request_tile<HD, kFBN>(Vs, p.v, b, hk, rank * kFBN, p.Sk, p.hd, p.vec);
  }
  for (int t = rank; t < tiles; t += nc) {
    const int key0 = t * kFBN, next0 = key0 + nc * kFBN;
    const bool more = t + nc < tiles;
    asm volatile("cp.async.wait_group 1;" ::: "memory");      // all but the V tile
    __syncthreads();
    float s[4][4];
    f32_tile_dot<HD>(Qs, Ks, ty, tx, s);
    __syncthreads();
    if (more) f32_request_tile<HD, kFBN>(Ks, p.k, b, hk, next0, p.Sk, p.hd, p.vec);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = row0 + ty * 4 + i;
      const int limit = p.causal ? min(p.Sk - 1, row + p.q_offset) : p.Sk - 1;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = key0 + tx + 16 * j <= limit ? s[i][j] * p.scale : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
      mx = fmaxf(m[i], half_warp_max(mx));
      const float sub = mx == -INFINITY ? 0.f : mx;
      const float alpha = expf(m[i] - sub);
      m[i] = mx;
      l[i] *= alpha;
#pragma unroll
      for (int c = 0; c < N; ++c) o[i][c] *= alpha;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = expf(s[i][j] - sub);
        l[i] += e;
        Ps[(ty * 4 + i) * LW + tx + 16 * j] = e;
      }
    }
    if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");      // all but the next K tile
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();       // (a row's weights are written and read by the same half warp)
    f32_tile_acc<HD>(Ps, Vs, ty, tx, o);
    __syncthreads();
    if (more) f32_request_tile<HD, kFBN>(Vs, p.v, b, hk, next0, p.Sk, p.hd, p.vec);
  }
  if constexpr (SHARED) {
    // Each CTA leaves its weighted sums, maxima and sums in shared memory (the tiles are idle by now); every one finishes an equal share
    // of the rows, in the order of the CTAs.
    cg::cluster_group cluster = cg::this_cluster();
    float* Os = Ks;                    // [kFBM][LD]
    float* Ms = Os + kFBM * LD;        // [kFBM] maximum, [kFBM] sum
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty * 4 + i;
#pragma unroll
      for (int c = 0; c < N; ++c) Os[r * LD + f32_col<HD>(tx, c)] = o[i][c];
      const float sum = half_warp_sum(l[i]);
      if (tx == 0) {
        Ms[r] = m[i];
        Ms[kFBM + r] = sum;
      }
    }
    cluster_sync_all();
    for (int i = rank * kFThreads + threadIdx.x; i < kFBM * HD; i += nc * kFThreads) {
      const int r = i / HD, d = i % HD, row = row0 + r;
      if (row >= p.Sq || d >= p.hd) continue;
      float mx = -INFINITY, x = 0.f, sum = 0.f;
      for (int c = 0; c < nc; ++c) mx = fmaxf(mx, cluster.map_shared_rank(Ms, c)[r]);
      const float sub = mx == -INFINITY ? 0.f : mx;
      for (int c = 0; c < nc; ++c) {
        const float w = expf(cluster.map_shared_rank(Ms, c)[r] - sub);
        x = fmaf(w, cluster.map_shared_rank(Os, c)[r * LD + d], x);
        sum = fmaf(w, cluster.map_shared_rank(Ms, c)[kFBM + r], sum);
      }
      p.o.p[b * p.o.sb + row * p.o.ss + h * p.o.sh + d] = x * (1.f / sum);
      if (p.lse && d == 0) p.lse[((long long)b * p.Hq + h) * p.Sq + row] = mx + logf(sum);
    }
    cluster_sync_all();                // nobody leaves while its shared memory is being read
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + ty * 4 + i;
    const float sum = half_warp_sum(l[i]);
    if (row >= p.Sq) continue;
    const float inv = 1.f / sum;      // nothing but -inf scores: NaN, as softmax has it
    float* dst = p.o.p + b * p.o.sb + row * p.o.ss + h * p.o.sh;
#pragma unroll
    for (int c = 0; c < N; ++c)
      if (f32_col<HD>(tx, c) < p.hd) dst[f32_col<HD>(tx, c)] = o[i][c] * inv;
    if (p.lse && tx == 0) p.lse[((long long)b * p.Hq + h) * p.Sq + row] = m[i] + logf(sum);
  }
}

// ---------------------------------------------------------------------------------------------------------------- decode
constexpr int kFDecRows = 8;      // query rows (group x Sq) of one kv head
template <int HD>
__global__ void __launch_bounds__(kFThreads)
attn_f32_decode(const AttnF32Params p) {
  constexpr int LD = f32_ld<HD>(), R = kFDecRows, LW = kFBN + 4;
  constexpr int C4 = HD / 4, G = kFThreads / C4;        // 16-byte columns, key groups of the weighted sum
  extern __shared__ float4 sm4[];
  float* Qs = reinterpret_cast<float*>(sm4);            // [R][LD]
  float* Ks = Qs + R * LD;
  float* Vs = Ks + kFBN * LD;
  float* Ps = Vs + kFBN * LD;                           // [R][LW]
  float* Os = Ps + R * LW;                              // [R][LD]: this CTA's weighted sum, read by its cluster
  float* Ms = Os + R * LD;                              // [R] maximum, [R] sum
  float* Ls = Ms + R;
  cg::cluster_group cluster = cg::this_cluster();
  const int nc = cluster.num_blocks(), rank = cluster.block_rank();
  const int hk = blockIdx.y, b = blockIdx.z, g = p.Hq / p.Hkv, rows = g * p.Sq;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = (p.Sk + kFBN - 1) / kFBN;
  // With rows to append, those that the caches have are older than the kernel ahead (the projection): this CTA's first tile of them is
  // requested before the wait for it.
  const bool ahead = p.appended < p.Sk && rank < tiles;
  if (ahead) {
    f32_request_tile<HD, kFBN>(Ks, p.k, b, hk, rank * kFBN, p.appended, p.hd, p.vec);
    f32_request_tile<HD, kFBN>(Vs, p.v, b, hk, rank * kFBN, p.appended, p.hd, p.vec);
  }
  pdl_wait();
  pdl_launch_dependents();
  // row r: query head hk * g + r / Sq, position r % Sq
  for (int i = tid; i < R * HD; i += kFThreads) {
    const int r = i / HD, d = i % HD;
    Qs[r * LD + d] = r < rows && d < p.hd ? p.q.p[b * p.q.sb + (r % p.Sq) * p.q.ss + (hk * g + r / p.Sq) * p.q.sh + d] : 0.f;
  }
  if (tid < R) {
    Ms[tid] = -INFINITY;
    Ls[tid] = 0.f;
  }
  float acc[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
  const int c4 = tid % C4, kg = tid / C4;
  for (int t = rank; t < tiles; t += nc) {
    const int key0 = t * kFBN;
    if (ahead && t == rank) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
      __syncthreads();
      f32_load_tile<HD, kFBN>(Ks, p.k, b, hk, key0, p.appended, p.hd, p.vec);
      f32_load_tile<HD, kFBN>(Vs, p.v, b, hk, key0, p.appended, p.hd, p.vec);
    }
    __syncthreads();
    if (key0 + kFBN > p.appended && p.appended < p.Sk) {
      // A tile is one CTA's alone, so that one appends its rows.
      const int first = max(key0, p.appended), count = min(p.Sk, key0 + kFBN) - first;
      for (int i = tid; i < count * p.hd; i += kFThreads) {
        const int key = first + i / p.hd, d = i % p.hd;
        const float x = p.kn.p[b * p.kn.sb + (key - p.appended) * p.kn.ss + hk * p.kn.sh + d];
        const float y = p.vn.p[b * p.vn.sb + (key - p.appended) * p.vn.ss + hk * p.vn.sh + d];
        Ks[(key - key0) * LD + d] = x;
        Vs[(key - key0) * LD + d] = y;
        p.k.p[b * p.k.sb + key * p.k.ss + hk * p.k.sh + d] = x;
        p.v.p[b * p.v.sb + key * p.v.ss + hk * p.v.sh + d] = y;
      }
      __syncthreads();
    }
    // scores: two threads per key, alternate 16-byte pieces
    const int key = tid >> 1;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = 0.f;
#pragma unroll 2
    for (int d = (tid & 1) * 4; d < HD; d += 8) {
      const float4 x = *reinterpret_cast<const float4*>(Ks + key * LD + d);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r >= rows) break;
        const float4 y = *reinterpret_cast<const float4*>(Qs + r * LD + d);
        s[r] = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s[r]))));
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r >= rows) break;
      const float full = (s[r] + __shfl_xor_sync(0xffffffffu, s[r], 1)) * p.scale;
      const int limit = p.causal ? min(p.Sk - 1, r % p.Sq + p.q_offset) : p.Sk - 1;
      if ((tid & 1) == 0) Ps[r * LW + key] = key0 + key <= limit ? full : -INFINITY;
    }
    __syncthreads();
    // softmax of a row's 64 scores: one warp per row
    for (int r = warp; r < rows; r += kFThreads / 32) {
      const float a = Ps[r * LW + lane], c = Ps[r * LW + lane + 32], m0 = Ms[r];
      float mx = fmaxf(a, c);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      mx = fmaxf(mx, m0);
      const float sub = mx == -INFINITY ? 0.f : mx;
      const float ea = expf(a - sub), ec = expf(c - sub);
      float sum = ea + ec;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      Ps[r * LW + lane] = ea;
      Ps[r * LW + lane + 32] = ec;
      if (lane == 0) {
        const float alpha = expf(m0 - sub);
        Ps[r * LW + kFBN] = alpha;                       // the padding column carries the row's rescaling factor
        Ls[r] = Ls[r] * alpha + sum;
        Ms[r] = mx;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r >= rows) break;
      const float alpha = Ps[r * LW + kFBN];
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] *= alpha;
    }
    for (int k = kg; k < kFBN; k += G) {
      const float4 x = *reinterpret_cast<const float4*>(Vs + k * LD + c4 * 4);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r >= rows) break;
        const float w = Ps[r * LW + k];
        acc[r][0] = fmaf(w, x.x, acc[r][0]);
        acc[r][1] = fmaf(w, x.y, acc[r][1]);
        acc[r][2] = fmaf(w, x.z, acc[r][2]);
        acc[r][3] = fmaf(w, x.w, acc[r][3]);
      }
    }
  }
  // fold the key groups in order (the K and V tiles are idle by now), then the CTAs of the cluster in rank order
  __syncthreads();
  float* fold = Ks;                                      // [G][C4 * 4] per row: at most 128 x 4 floats
  for (int r = 0; r < rows; ++r) {
#pragma unroll
    for (int rr = 0; rr < R; ++rr)
      if (rr == r) *reinterpret_cast<float4*>(fold + tid * 4) = make_float4(acc[rr][0], acc[rr][1], acc[rr][2], acc[rr][3]);
    __syncthreads();
    for (int d = tid; d < HD; d += kFThreads) {
      float x = 0.f;
      for (int k = 0; k < G; ++k) x += fold[(k * C4 + d / 4) * 4 + d % 4];
      Os[r * LD + d] = x;
    }
    __syncthreads();
  }
  cluster_sync_all();
  for (int i = rank * kFThreads + tid; i < rows * p.hd; i += nc * kFThreads) {
    const int r = i / p.hd, d = i % p.hd;
    float mx = -INFINITY;
    for (int c = 0; c < nc; ++c) mx = fmaxf(mx, cluster.map_shared_rank(Ms, c)[r]);
    const float sub = mx == -INFINITY ? 0.f : mx;
    float x = 0.f, sum = 0.f;
    for (int c = 0; c < nc; ++c) {
      const float w = expf(cluster.map_shared_rank(Ms, c)[r] - sub);
      x = fmaf(w, cluster.map_shared_rank(Os, c)[r * LD + d], x);
      sum = fmaf(w, cluster.map_shared_rank(Ls, c)[r], sum);
    }
    const int row = r % p.Sq, h = hk * g + r / p.Sq;
    p.o.p[b * p.o.sb + row * p.o.ss + h * p.o.sh + d] = x / sum;
    if (p.lse && d == 0) p.lse[((long long)b * p.Hq + h) * p.Sq + row] = sub + logf(sum);
  }
  cluster_sync_all();      // nobody leaves while its shared memory is being read
}

// -------------------------------------------------------------------------------------------------------------- backward
// P and dS = scale * P * (dP - delta) of one 32 x 64 tile, rows against their statistics.
template <int HD>
__device__ __forceinline__ void f32_probs(const AttnF32Params& p, const float* Qs, const float* Ks, const float* dOs, const float* Vs,
                                          int row0, int key0, int ty, int tx, const float (&lse)[4], const float (&delta)[4],
                                          float (&pr)[4][4], float (&ds)[4][4]) {
  f32_tile_dot<HD>(Qs, Ks, ty, tx, pr);
  f32_tile_dot<HD>(dOs, Vs, ty, tx, ds);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + ty * 4 + i;
    const int limit = row >= p.Sq ? -1 : p.causal ? min(p.Sk - 1, row + p.q_offset) : p.Sk - 1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool seen = key0 + tx + 16 * j <= limit;
      pr[i][j] = seen ? expf(pr[i][j] * p.scale - lse[i]) : 0.f;
      ds[i][j] = seen ? pr[i][j] * (ds[i][j] - delta[i]) * p.scale : 0.f;
    }
  }
}

template <int HD>
__global__ void __launch_bounds__(kFThreads)
attn_f32_dq(const AttnF32Params p) {
  extern __shared__ float4 sm4[];
  constexpr int LD = f32_ld<HD>(), LW = kFBN + 4, N = F32Cols<HD>::N;
  float* Qs = reinterpret_cast<float*>(sm4);
  float* dOs = Qs + kFBM * LD;
  float* Ks = dOs + kFBM * LD;
  float* Vs = Ks + kFBN * LD;
  float* dSs = Vs + kFBN * LD;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // As in the forward, and in attn_f32_dkv: by length, over all heads.  (B200, causal, forward and backward together, all three so: 4 x
  // 700 tokens of 8 heads of 64 496 -> 407 us, 16 x 200 of 6 heads 198 -> 155, 8 x 128 of 8 heads of 32 46.8 -> 44.6 us.)
  const int qx = blockIdx.x / (p.B * p.Hq), bh = blockIdx.x - qx * p.B * p.Hq;
  const int qt = p.causal ? (p.Sq + kFBM - 1) / kFBM - 1 - qx : qx;
  const int b = bh / p.Hq, h = bh - b * p.Hq, hk = h / (p.Hq / p.Hkv), row0 = qt * kFBM;
  f32_load_tile<HD, kFBM>(Qs, p.q, b, h, row0, p.Sq, p.hd, p.vec);
  f32_load_tile<HD, kFBM>(dOs, p.dout, b, h, row0, p.Sq, p.hd, p.vec);
  f32_load_tile<HD, kFBM>(Ks, p.o, b, h, row0, p.Sq, p.hd, p.vec);      // O, before the first keys
  __syncthreads();
  float lse[4], delta[4], dq[4][N];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i, row = row0 + r;
    const long long at = ((long long)b * p.Hq + h) * p.Sq + row;
    float x = 0.f;
#pragma unroll
    for (int c = 0; c < N; ++c) x = fmaf(dOs[r * LD + tx * N + c], Ks[r * LD + tx * N + c], x);
    delta[i] = half_warp_sum(x);
    lse[i] = row < p.Sq ? p.lse[at] : 0.f;
    if (row < p.Sq && tx == 0) p.delta[at] = delta[i];
#pragma unroll
    for (int c = 0; c < N; ++c) dq[i][c] = 0.f;
  }
  const int tiles = f32_key_tiles(p, row0);
  for (int t = 0; t < tiles; ++t) {
    const int key0 = t * kFBN;
    __syncthreads();
    f32_load_tile<HD, kFBN>(Ks, p.k, b, hk, key0, p.Sk, p.hd, p.vec);
    f32_load_tile<HD, kFBN>(Vs, p.v, b, hk, key0, p.Sk, p.hd, p.vec);
    __syncthreads();
    float pr[4][4], ds[4][4];
    f32_probs<HD>(p, Qs, Ks, dOs, Vs, row0, key0, ty, tx, lse, delta, pr, ds);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dSs[(ty * 4 + i) * LW + tx + 16 * j] = ds[i][j];
    __syncwarp();
    f32_tile_acc<HD>(dSs, Ks, ty, tx, dq);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + ty * 4 + i;
    if (row >= p.Sq) continue;
    float* dst = p.dq.p + b * p.dq.sb + row * p.dq.ss + h * p.dq.sh;
#pragma unroll
    for (int c = 0; c < N; ++c)
      if (f32_col<HD>(tx, c) < p.hd) dst[f32_col<HD>(tx, c)] = dq[i][c];
  }
}

// out[i][c] += sum over 32 rows of W[row][ty * 8 + i] * X[row][column c of this thread]
template <int HD>
__device__ __forceinline__ void f32_tile_acc_t(const float* W, const float* X, int ty, int tx, float (&out)[8][F32Cols<HD>::N]) {
  constexpr int LD = f32_ld<HD>(), N = F32Cols<HD>::N, RUN = F32Cols<HD>::RUN, LW = kFBN + 4;
#pragma unroll 4
  for (int r = 0; r < kFBM; ++r) {
    const float4 w0 = *reinterpret_cast<const float4*>(W + r * LW + ty * 8);
    const float4 w1 = *reinterpret_cast<const float4*>(W + r * LW + ty * 8 + 4);
    const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int c = 0; c < N; c += RUN) {
      const float* src = X + r * LD + f32_col<HD>(tx, c);
      float v[RUN];
      if constexpr (RUN == 4) {
        const float4 x = *reinterpret_cast<const float4*>(src);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
      } else if constexpr (RUN == 2) {
        const float2 x = *reinterpret_cast<const float2*>(src);
        v[0] = x.x; v[1] = x.y;
      } else {
        v[0] = *src;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < RUN; ++e) out[i][c + e] = fmaf(w[i], v[e], out[i][c + e]);
    }
  }
}

template <int HD>
__global__ void __launch_bounds__(kFThreads)
attn_f32_dkv(const AttnF32Params p) {
  extern __shared__ float4 sm4[];
  constexpr int LD = f32_ld<HD>(), LW = kFBN + 4, N = F32Cols<HD>::N;
  float* Qs = reinterpret_cast<float*>(sm4);
  float* dOs = Qs + kFBM * LD;
  float* Ks = dOs + kFBM * LD;
  float* Vs = Ks + kFBN * LD;
  float* Ps = Vs + kFBN * LD;
  float* dSs = Ps + kFBM * LW;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int kt = blockIdx.x / (p.B * p.Hkv), bh = blockIdx.x - kt * p.B * p.Hkv;    // (causal: the first keys see the most rows)
  const int b = bh / p.Hkv, hk = bh - b * p.Hkv, g = p.Hq / p.Hkv, key0 = kt * kFBN;
  f32_load_tile<HD, kFBN>(Ks, p.k, b, hk, key0, p.Sk, p.hd, p.vec);
  f32_load_tile<HD, kFBN>(Vs, p.v, b, hk, key0, p.Sk, p.hd, p.vec);
  float dk[8][N], dv[8][N];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < N; ++c) dk[i][c] = dv[i][c] = 0.f;
  const int first = p.causal ? max(0, key0 - p.q_offset) / kFBM : 0;     // first row tile that sees a key of this tile
  const int row_tiles = (p.Sq + kFBM - 1) / kFBM;
  for (int e = 0; e < g; ++e) {
    const int h = hk * g + e;
    for (int t = first; t < row_tiles; ++t) {
      const int row0 = t * kFBM;
      __syncthreads();
      f32_load_tile<HD, kFBM>(Qs, p.q, b, h, row0, p.Sq, p.hd, p.vec);
      f32_load_tile<HD, kFBM>(dOs, p.dout, b, h, row0, p.Sq, p.hd, p.vec);
      float lse[4], delta[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = row0 + ty * 4 + i;
        const long long at = ((long long)b * p.Hq + h) * p.Sq + min(row, p.Sq - 1);
        lse[i] = p.lse[at];
        delta[i] = p.delta[at];
      }
      __syncthreads();
      float pr[4][4], ds[4][4];
      f32_probs<HD>(p, Qs, Ks, dOs, Vs, row0, key0, ty, tx, lse, delta, pr, ds);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          Ps[(ty * 4 + i) * LW + tx + 16 * j] = pr[i][j];
          dSs[(ty * 4 + i) * LW + tx + 16 * j] = ds[i][j];
        }
      __syncthreads();
      f32_tile_acc_t<HD>(Ps, dOs, ty, tx, dv);
      f32_tile_acc_t<HD>(dSs, Qs, ty, tx, dk);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int key = key0 + ty * 8 + i;
    if (key >= p.Sk) continue;
    float* dkp = p.dk.p + b * p.dk.sb + key * p.dk.ss + hk * p.dk.sh;
    float* dvp = p.dv.p + b * p.dv.sb + key * p.dv.ss + hk * p.dv.sh;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const int d = f32_col<HD>(tx, c);
      if (d < p.hd) {
        dkp[d] = dk[i][c];
        dvp[d] = dv[i][c];
      }
    }
  }
}

template <int HD> constexpr int f32_smem(int hd_rows, int w_rows) {
  return (hd_rows * f32_ld<HD>() + w_rows * (kFBN + 4)) * 4;
}

// CTAs for the keys of a row tile: 1, 2 or 4, by what the longest rows weigh in even shares of the key tiles (see the launch).
static int f32_key_ctas(const AttnF32Params& p, bool wide) {
  const int qtiles = (p.Sq + kFBM - 1) / kFBM, longest = f32_key_tiles(p, (qtiles - 1) * kFBM);
  const long long heads = (long long)p.Hq * p.B, room = (long long)longest * sm_count();
  if (longest < 4 || heads * qtiles > room) return 1;
  long long work = 0;
  for (int t = 0; t < qtiles; ++t) work += heads * f32_key_tiles(p, t * kFBM);
  if (room >= 2 * work) return 4;
  return longest >= 8 && (wide ? 4 * room >= 5 * work : room >= work) ? 2 : 1;
}

template <int HD>
static int attn_f32_launch(const AttnF32Params& p, int backward, cudaStream_t st) {
  const dim3 qgrid((p.Sq + kFBM - 1) / kFBM, p.Hq, p.B);
  if (!backward) {
    // Few rows of a kv head (decoding): the keys are split over a cluster, one 64-key tile and up for each CTA.  GPT-2 124M,
    // one row over 510 keys: 12 CTAs of the tile kernel against 96 here.
    if (p.Hq / p.Hkv * p.Sq <= kFDecRows) {
      const int smem = f32_smem<HD>(2 * kFBN + 2 * kFDecRows, kFDecRows) + 2 * kFDecRows * 4;
      const int tiles = (p.Sk + kFBN - 1) / kFBN;
      int nc = 1;
      while (nc < 8 && nc < tiles) nc *= 2;
      DPTB_CUDA_OK(cudaFuncSetAttribute(attn_f32_decode<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(nc, p.Hkv, p.B);
      cfg.blockDim = dim3(kFThreads);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = st;
      cudaLaunchAttribute at[2];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = nc;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.numAttrs = pdl_flag() ? 2 : 1;
      return counted(1, (int)cudaLaunchKernelEx(&cfg, attn_f32_decode<HD>, p));
    }
    const int smem = f32_smem<HD>(kFBM + 2 * kFBN, kFBM);
    // The time of a launch is that of the SM with the most key tiles: one CTA keeps an SM's shared memory busy, two at once take twice as
    // long (3.1 us a tile at heads of 64).  Where the longest rows weigh as much as an SM's even share of the tiles, two CTAs divide
    // them, and four where they weigh twice as much; each CTA more costs 2 to 3 us of meeting, so that shorter rows stay whole.  B200,
    // one / two / four CTAs, causal: 12 heads of 64, 509 tokens 31.1 / 28.5 / 32.2 us (longest rows 1.4 even shares), 256 tokens
    // 16.0 / 17.3 / 14.2 (2.5), 2 x 512 tokens 43.0 / 47.9 / 52.2 (0.7); 8 heads of 32, 512 tokens 19.7 / 16.4 / 13.6 (2.1); heads of
    // 128, of which an SM holds two: 2 heads, 1024 tokens 92.4 / 58.8 / 38.8 (4.3), 10 heads, 512 tokens 51.6 / 46.6 / 58.5 (1.6),
    // 16 heads 60.4 / 70.2 / 85.0 (1.0).
    AttnF32Params s = p;
    s.key_ctas = f32_key_ctas(p, HD > 64);
    const long long ctas = (long long)qgrid.x * qgrid.y * qgrid.z;
    const dim3 grid((unsigned)(ctas * s.key_ctas));
    if (s.key_ctas == 1) {
      DPTB_CUDA_OK(cudaFuncSetAttribute(attn_f32_fwd<HD, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      return counted(1, (int)launch_k(attn_f32_fwd<HD, false>, grid, dim3(kFThreads), (size_t)smem, st, s));
    }
    DPTB_CUDA_OK(cudaFuncSetAttribute(attn_f32_fwd<HD, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kFThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = s.key_ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl_flag() ? 2 : 1;
    return counted(1, (int)cudaLaunchKernelEx(&cfg, attn_f32_fwd<HD, true>, s));
  }
  const int smem_q = f32_smem<HD>(2 * kFBM + 2 * kFBN, kFBM), smem_kv = f32_smem<HD>(2 * kFBM + 2 * kFBN, 2 * kFBM);
  DPTB_CUDA_OK(cudaFuncSetAttribute(attn_f32_dq<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_q));
  DPTB_CUDA_OK(cudaFuncSetAttribute(attn_f32_dkv<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_kv));
  attn_f32_dq<HD><<<dim3(qgrid.x * qgrid.y * qgrid.z), kFThreads, smem_q, st>>>(p);
  DPTB_CUDA_OK(cudaGetLastError());
  attn_f32_dkv<HD><<<dim3((unsigned)((p.Sk + kFBN - 1) / kFBN) * p.Hkv * p.B), kFThreads, smem_kv, st>>>(p);
  return counted(2, (int)cudaGetLastError());
}

}  // namespace dptb

using namespace dptb;

static int attn_f32(const DptbAttnF32Args* a, const DptbF32View* kn, const DptbF32View* vn, void* stream) {
  if (a->B <= 0 || a->Sq <= 0 || a->Hq <= 0) return 0;
  if (a->hd <= 0 || a->hd > 128) return kErrUnsupported;
  if (a->Sk <= 0 || a->Hkv <= 0 || a->Hq % a->Hkv || a->q_offset < 0) return kErrBadShape;
  if (a->B > 65535 || a->Hq > 65535) return kErrTooLarge;
  if (a->backward && (!a->lse || !a->delta)) return kErrBadShape;
  AttnF32Params p;
  p.vec = a->hd % 4 == 0;
  const DptbF32View* in[8] = {&a->q, &a->k, &a->v, &a->o, &a->dout, &a->dq, &a->dk, &a->dv};
  F32View* out[8] = {&p.q, &p.k, &p.v, &p.o, &p.dout, &p.dq, &p.dk, &p.dv};
  for (int i = 0; i < 8; ++i) {
    *out[i] = F32View{in[i]->p, in[i]->sb, in[i]->ss, in[i]->sh};
    if (i >= 4 && !a->backward) continue;
    if (!in[i]->p) return kErrBadShape;
    if ((reinterpret_cast<uintptr_t>(in[i]->p) & 15) || (in[i]->sb | in[i]->ss | in[i]->sh) % 4) p.vec = 0;
  }
  p.kn = kn ? F32View{kn->p, kn->sb, kn->ss, kn->sh} : F32View{};
  p.vn = vn ? F32View{vn->p, vn->sb, vn->ss, vn->sh} : F32View{};
  p.appended = kn ? a->Sk - a->Sq : a->Sk;
  p.key_ctas = 1;
  p.lse = a->lse;
  p.delta = a->delta;
  p.B = a->B; p.Sq = a->Sq; p.Sk = a->Sk; p.Hq = a->Hq; p.Hkv = a->Hkv; p.hd = a->hd;
  p.causal = a->causal;
  p.q_offset = a->q_offset;
  p.scale = a->scale;
  auto st = static_cast<cudaStream_t>(stream);
  if (a->hd <= 16) return attn_f32_launch<16>(p, a->backward, st);
  if (a->hd <= 32) return attn_f32_launch<32>(p, a->backward, st);
  if (a->hd <= 64) return attn_f32_launch<64>(p, a->backward, st);
  return attn_f32_launch<128>(p, a->backward, st);
}
extern "C" int dptb_attn_f32(const DptbAttnF32Args* a, void* stream) { return attn_f32(a, nullptr, nullptr, stream); }

// Decoding with the cache append in the same kernel: k and v are caches, the last Sq of their Sk rows come from kn and vn.  A step of few
// rows is a chain of short kernels: GPT-2 124M, one token over 509, spent 3.5 us a layer in the copy alone.  kErrUnsupported where the
// rows are too many for the decode kernel: the caller appends, then attends.
extern "C" int dptb_attn_f32_append(const DptbAttnF32Args* a, const DptbF32View* kn, const DptbF32View* vn, void* stream) {
  if (a->backward || a->Hkv <= 0 || a->Hq % a->Hkv || a->Hq / a->Hkv * a->Sq > kFDecRows || a->Sk < a->Sq || !kn->p || !vn->p)
    return kErrUnsupported;
  return attn_f32(a, kn, vn, stream);
}
