// Embedding gather (optionally fused with a learned position table) and its scatter-add backward.
//
// Out-of-range indices read as a zero row and are skipped in the backward, as in the reference
// (lib/native/src/kernels/embedding.cuh:19-48).  The backward comes in three forms: a sorted,
// segmented sum (one warp per distinct index, rows added in ascending order -> bit-reproducible), a form
// for short index lists that finds the equal indices itself instead of having them sorted (the same additions in the same
// order), and an atomic form.
#include "common/host.h"
#include "common/reduce.cuh"

namespace dptb {

// out[n, :] = table[idx[n], :] (+ pos_table[(pos_start + n % seq_len), :]).  One warp per row.
template <typename T>
__global__ void __launch_bounds__(256)
embedding_fwd_kernel(const T* __restrict__ table, long long vocab, const long long* __restrict__ idx,
                     const T* __restrict__ pos_table, long long pos_rows, int pos_start, int seq_len,
                     T* __restrict__ out, long long n, int D, int vec_ok) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r = warp0; r < n; r += nwarps) {
    const long long t = idx[r];
    const bool ok = t >= 0 && t < vocab;
    const long long ppos = pos_table ? (long long)pos_start + (seq_len > 0 ? r % seq_len : r) : 0;
    const bool pok = pos_table && ppos >= 0 && ppos < pos_rows;
    const T* src = table + (ok ? t : 0) * D;
    const T* psrc = pos_table ? pos_table + (pok ? ppos : 0) * D : nullptr;
    T* dst = out + r * D;
    if (vec_ok) {
      for (int c = lane * 8; c < D; c += 256) {
        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (ok) Vec8<T>::load(src + c, v);
        if (pok) {
          float pv[8];
          Vec8<T>::load(psrc + c, pv);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] += pv[j];
        }
        Vec8<T>::store(dst + c, v);
      }
    } else {
      for (int c = lane; c < D; c += 32) {
        float v = ok ? to_f32(src[c]) : 0.0f;
        if (pok) v += to_f32(psrc[c]);
        dst[c] = from_f32<T>(v);
      }
    }
  }
}

__device__ __forceinline__ void atomic_add_t(float* p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_t(__nv_bfloat16* p, float v) { atomicAdd(p, __float2bfloat16(v)); }

// dtable[idx[n], :] += dout[n, :] with atomics (order of equal indices not fixed).
template <typename T>
__global__ void __launch_bounds__(256)
embedding_bwd_atomic_kernel(T* __restrict__ dtable, long long vocab, const long long* __restrict__ idx,
                            const T* __restrict__ dout, long long n, int D) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r = warp0; r < n; r += nwarps) {
    const long long t = idx[r];
    if (t < 0 || t >= vocab) continue;
    for (int c = lane; c < D; c += 32) atomic_add_t(dtable + t * D + c, to_f32(dout[r * D + c]));
  }
}

// Sorted form: sorted_idx ascending, perm[i] = source row of sorted position i (stable order).  The warp that sits on
// the first position of a run of equal indices adds the whole run in order and does one read-modify-write.
template <typename T>
__global__ void __launch_bounds__(256)
embedding_bwd_sorted_kernel(T* __restrict__ dtable, long long vocab, const long long* __restrict__ sorted_idx,
                            const long long* __restrict__ perm, const T* __restrict__ dout, long long n, int D,
                            int vec_ok) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long i = warp0; i < n; i += nwarps) {
    const long long t = sorted_idx[i];
    if (t < 0 || t >= vocab) continue;
    if (i > 0 && sorted_idx[i - 1] == t) continue;  // not a run start
    long long end = i + 1;
    while (end < n && sorted_idx[end] == t) ++end;
    if (vec_ok) {
      // 16-byte accesses: a lane owns 8 consecutive features of the row, rows of the run are added in order
      for (int c = lane * 8; c < D; c += 256) {
        float acc[8];
        Vec8<T>::load(dtable + t * D + c, acc);
        for (long long k = i; k < end; ++k) {
          float v[8];
          Vec8<T>::load(dout + perm[k] * D + c, v);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[j] += v[j];
        }
        Vec8<T>::store(dtable + t * D + c, acc);
      }
    } else {
      for (int c = lane; c < D; c += 32) {
        float acc = to_f32(dtable[t * D + c]);
        for (long long k = i; k < end; ++k) acc += to_f32(dout[perm[k] * D + c]);
        dtable[t * D + c] = from_f32<T>(acc);
      }
    }
  }
}

// Short lists, unsorted: the warp of the first token with an index adds all later ones in order.  The list is held in shared
// memory (32 keys a step, compared by ballot), blockIdx.y takes 256 features; up to four rows are loaded before they are added.
// A sort of the list costs 25 us and more whatever its length.  Measured (B200, whole backward, against the one with the
// sort): 603 tokens of 128 features 6.3 us, 33 us with it; 1024 tokens over 65 indices, 256 features, 12 and 38 us;
// 2048 tokens over 50257 indices, 768 features, 13 and 35 us;
// 4096 of them 39 and 42 us, 8192 131 and 104 us, so lists stop at 2048.
template <typename T>
__global__ void __launch_bounds__(256)
embedding_bwd_scan_kernel(T* __restrict__ dtable, int vocab, const long long* __restrict__ idx, const T* __restrict__ dout,
                          int n, int D, int vec_ok) {
  extern __shared__ int keys[];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const long long t = idx[i];
    keys[i] = t >= 0 && t < vocab ? (int)t : -1;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const int t = keys[i];
  if (t < 0) return;
  for (int hi = i; hi > 0; hi -= 32) {                 // an earlier token with this index?
    const int j = hi - 1 - lane;
    if (__any_sync(0xffffffffu, j >= 0 && keys[j] == t)) return;
  }
  const int c0 = blockIdx.y * 256;
  T* row = dtable + (long long)t * D;
  if (vec_ok) {
    const int c = c0 + lane * 8;
    const bool live = c < D;
    float acc[8];
    if (live) Vec8<T>::load(row + c, acc);
    for (int base = i; base < n; base += 32) {
      unsigned mask = __ballot_sync(0xffffffffu, base + lane < n && keys[base + lane] == t);
      while (mask) {
        Raw8<T> v[4];
        int m = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (mask) {
            const int j = base + __ffs(mask) - 1;
            mask &= mask - 1;
            if (live) v[u].load(dout + (long long)j * D + c);
            m = u + 1;
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (live && u < m) {
            float f[8];
            v[u].unpack(f);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += f[k];
          }
      }
    }
    if (live) Vec8<T>::store(row + c, acc);
  } else {
    const int c1 = min(D, c0 + 256);
    for (int cw = c0; cw < c1; cw += 32) {             // whole warps reach the ballot
      const int c = cw + lane;
      const bool live = c < c1;
      float acc = live ? to_f32(row[c]) : 0.0f;
      for (int base = i; base < n; base += 32) {
        unsigned mask = __ballot_sync(0xffffffffu, base + lane < n && keys[base + lane] == t);
        for (; mask; mask &= mask - 1)
          if (live) acc += to_f32(dout[(long long)(base + __ffs(mask) - 1) * D + c]);
      }
      if (live) row[c] = from_f32<T>(acc);
    }
  }
}

// Learned positions are an arange, so their gradient is a strided batch sum: dpos[p, :] += sum_b dout[b*S + (p - start), :].
template <typename T>
__global__ void __launch_bounds__(256)
pos_embedding_bwd_kernel(T* __restrict__ dpos, long long pos_rows, int pos_start, int seq_len, long long batch,
                         const T* __restrict__ dout, int D) {
  const long long total = (long long)seq_len * D;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const long long s = e / D;
    const int c = (int)(e % D);
    const long long p = s + pos_start;
    if (p < 0 || p >= pos_rows) continue;
    float acc = to_f32(dpos[p * D + c]);
    for (long long b = 0; b < batch; ++b) acc += to_f32(dout[(b * seq_len + s) * D + c]);
    dpos[p * D + c] = from_f32<T>(acc);
  }
}

static inline int warp_grid(long long n) {
  long long blocks = (n + 7) / 8;
  const long long cap = (long long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  return (int)(blocks < 1 ? 1 : blocks);
}

}  // namespace dptb

using namespace dptb;

extern "C" int dptb_embedding_fwd(const void* table, long long vocab, const long long* idx, const void* pos_table,
                                  long long pos_rows, int pos_start, int seq_len, void* out, long long n, int D,
                                  int dtype, void* stream) {
  if (n <= 0) return 0;
  auto st = static_cast<cudaStream_t>(stream);
  const int vec_ok = (D % 8 == 0) && (((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(pos_table) |
                                        reinterpret_cast<uintptr_t>(out)) & 15) == 0);
  if (dtype) embedding_fwd_kernel<__nv_bfloat16><<<warp_grid(n), 256, 0, st>>>((const __nv_bfloat16*)table, vocab, idx, (const __nv_bfloat16*)pos_table, pos_rows, pos_start, seq_len, (__nv_bfloat16*)out, n, D, vec_ok);
  else       embedding_fwd_kernel<float><<<warp_grid(n), 256, 0, st>>>((const float*)table, vocab, idx, (const float*)pos_table, pos_rows, pos_start, seq_len, (float*)out, n, D, vec_ok);
  return counted(1, (int)cudaGetLastError());
}
// The list as it is, at most kScanTokens long.
constexpr int kScanTokens = 2048;
extern "C" int dptb_embedding_bwd_scan(void* dtable, long long vocab, const long long* idx, const void* dout, long long n, int D,
                                       int dtype, void* stream) {
  if (n <= 0 || D <= 0) return 0;
  if (n > kScanTokens || vocab > 0x7fffffffLL || D > 256 * 65535) return kErrTooLarge;
  auto st = static_cast<cudaStream_t>(stream);
  const int vec_ok = (D % 8 == 0) && (((reinterpret_cast<uintptr_t>(dtable) | reinterpret_cast<uintptr_t>(dout)) & 15) == 0);
  const dim3 grid((unsigned)((n + 7) / 8), (unsigned)((D + 255) / 256));
  const size_t smem = (size_t)n * 4;
  if (dtype) embedding_bwd_scan_kernel<__nv_bfloat16><<<grid, 256, smem, st>>>((__nv_bfloat16*)dtable, (int)vocab, idx, (const __nv_bfloat16*)dout, (int)n, D, vec_ok);
  else       embedding_bwd_scan_kernel<float><<<grid, 256, smem, st>>>((float*)dtable, (int)vocab, idx, (const float*)dout, (int)n, D, vec_ok);
  return counted(1, (int)cudaGetLastError());
}
// sorted_idx / perm may be null: then the atomic form runs.
extern "C" int dptb_embedding_bwd(void* dtable, long long vocab, const long long* idx, const long long* sorted_idx,
                                  const long long* perm, const void* dout, long long n, int D, int dtype, void* stream) {
  if (n <= 0) return 0;
  auto st = static_cast<cudaStream_t>(stream);
  if (sorted_idx && perm) {
    const int vec_ok = (D % 8 == 0) && (((reinterpret_cast<uintptr_t>(dtable) | reinterpret_cast<uintptr_t>(dout)) & 15) == 0);
    if (dtype) embedding_bwd_sorted_kernel<__nv_bfloat16><<<warp_grid(n), 256, 0, st>>>((__nv_bfloat16*)dtable, vocab, sorted_idx, perm, (const __nv_bfloat16*)dout, n, D, vec_ok);
    else       embedding_bwd_sorted_kernel<float><<<warp_grid(n), 256, 0, st>>>((float*)dtable, vocab, sorted_idx, perm, (const float*)dout, n, D, vec_ok);
  } else {
    if (dtype) embedding_bwd_atomic_kernel<__nv_bfloat16><<<warp_grid(n), 256, 0, st>>>((__nv_bfloat16*)dtable, vocab, idx, (const __nv_bfloat16*)dout, n, D);
    else       embedding_bwd_atomic_kernel<float><<<warp_grid(n), 256, 0, st>>>((float*)dtable, vocab, idx, (const float*)dout, n, D);
  }
  return counted(1, (int)cudaGetLastError());
}
extern "C" int dptb_pos_embedding_bwd(void* dpos, long long pos_rows, int pos_start, int seq_len, long long batch,
                                      const void* dout, int D, int dtype, void* stream) {
  if (seq_len <= 0 || batch <= 0) return 0;
  auto st = static_cast<cudaStream_t>(stream);
  const long long total = (long long)seq_len * D;
  int blocks = (int)((total + 255) / 256);
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  if (dtype) pos_embedding_bwd_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>((__nv_bfloat16*)dpos, pos_rows, pos_start, seq_len, batch, (const __nv_bfloat16*)dout, D);
  else       pos_embedding_bwd_kernel<float><<<blocks, 256, 0, st>>>((float*)dpos, pos_rows, pos_start, seq_len, batch, (const float*)dout, D);
  return counted(1, (int)cudaGetLastError());
}
