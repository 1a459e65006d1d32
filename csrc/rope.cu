// Rotary embedding on the head blocks of token rows, and its fusion with the append to a key / value cache.
//
// Half-split form: element (t, h, d) sits at x[t * ld + h * head_dim + d]; for d < rotary_dim / 2 the pair (d, d + rotary_dim / 2)
// is turned by pos * base^(-2 d / rotary_dim), the dimensions from rotary_dim on pass through
// (reference: lib/core/nn/rotary.dart:95-201).  The position of token t is positions[t] when given, else
// pos_start + (t % seq_len); `inverse` turns the other way (the backward).
//
// With a cache the row is [Hq | Hkv | Hkv] heads: the queries are turned in place, the keys are turned on their way into the
// cache and the values copied there, so a projection's output is read once and no copy kernels follow
// (reference: lib/core/nn/kv_cache.dart:22-84 concatenates through the host).
//
// A block takes up to 8 tokens and computes their angles once into shared memory, one accurate power, sine and cosine per
// (token, pair) instead of one per element; the heads then go by in 16-byte groups.  Bound by memory.  Measured (B200),
// 6124 tokens x 20 heads of 64 in bf16, in place: one angle per element 40 us, this 9.2 us; 8192 tokens x 20 heads of 128: 100 us -> 18 us.
#include "common/host.h"
#include "common/reduce.cuh"

namespace dptb {

constexpr int kRopeThreads = 256;
constexpr int kRopeTokens = 8;
constexpr int kRopeTable = 2048;   // angles held at a time

struct RopeParams {
  const void* x;
  void* out;
  long long tokens, ld_in, ld_out;
  int heads, head_dim, rotary_dim, seq_len, pos_start, inverse;
  float base;
  const long long* positions;
  int tokens_per_block;
  // cache form: kc != nullptr
  void* kc;
  void* vc;
  long long ldkv, kv_batch_stride;
  int kv_heads, row0, cap;   // token s of a sequence goes to cache row row0 + s; none at or beyond cap is written
  const int* pos_ptr;        // when set: pos_start and row0 both come from here
};

template <typename T, int VEC>
struct RopeVec;
template <typename T>
struct RopeVec<T, 1> {
  static __device__ __forceinline__ void load(const T* p, float (&v)[1]) { v[0] = to_f32(*p); }
  static __device__ __forceinline__ void store(T* p, const float (&v)[1]) { *p = from_f32<T>(v[0]); }
};
template <>
struct RopeVec<float, 4> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct RopeVec<__nv_bfloat16, 8> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[8]) { Vec8<__nv_bfloat16>::load(p, v); }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[8]) { Vec8<__nv_bfloat16>::store(p, v); }
};

template <typename T, int VEC>
__global__ void __launch_bounds__(kRopeThreads)
rope_kernel(const RopeParams p) {
  // As a programmatic dependent the first angles are worked out before the kernel ahead is done, unless positions come from the device.
  bool waits = !p.pos_ptr && !p.positions;
  auto wait = [&] {
    pdl_wait();              // (no-ops in an ordinary launch)
    pdl_launch_dependents();
  };
  if (!waits) wait();
  __shared__ float2 table[kRopeTable];
  using V = RopeVec<T, VEC>;
  const long long t0 = (long long)blockIdx.x * p.tokens_per_block;
  const int nt = (int)min((long long)p.tokens_per_block, p.tokens - t0);
  const int half = p.rotary_dim / 2;
  const int pos_start = p.pos_ptr ? *p.pos_ptr : p.pos_start;
  const int row0 = p.pos_ptr ? pos_start : p.row0;
  const bool cache = p.kc != nullptr;
  const int kv = cache ? p.kv_heads : 0;
  const T* x = static_cast<const T*>(p.x);
  T* out = static_cast<T*>(p.out);

  // Where element (t, h, 0) goes, or null when it has no place in the cache.
  auto dest = [&](int t, int h) -> T* {
    const long long tok = t0 + t;
    if (!cache) return out + tok * p.ld_out + (long long)h * p.head_dim;
    const long long b = tok / p.seq_len;
    const long long row = row0 + tok % p.seq_len;
    if (row >= p.cap) return nullptr;
    if (h < p.heads) return out + tok * p.ld_out + (long long)h * p.head_dim;
    const bool is_v = h >= p.heads + kv;
    return static_cast<T*>(is_v ? p.vc : p.kc) + b * p.kv_batch_stride + row * p.ldkv +
           (long long)(h - p.heads - (is_v ? kv : 0)) * p.head_dim;
  };

  const int turned = p.heads + kv;
  const int chunk = min(half, kRopeTable / p.tokens_per_block / VEC * VEC);
  for (int d0 = 0; d0 < half; d0 += chunk) {
    const int n = min(chunk, half - d0);
    if (d0 > 0) __syncthreads();
    for (int i = threadIdx.x; i < nt * n; i += kRopeThreads) {
      const int t = i / n, d = d0 + i % n;
      const long long tok = t0 + t;
      const float pos = p.positions ? (float)p.positions[tok]
                                    : (float)(pos_start + (p.seq_len > 0 ? tok % p.seq_len : tok));
      const float inv = powf(p.base, -2.0f * (float)d / (float)p.rotary_dim);
      float sn, cs;
      sincosf(pos * inv, &sn, &cs);
      table[i] = make_float2(cs, p.inverse ? -sn : sn);
    }
    if (waits) wait();
    waits = false;
    __syncthreads();
    const int groups = n / VEC, per_tok = turned * groups;
    for (int i = threadIdx.x; i < nt * per_tok; i += kRopeThreads) {
      const int t = i / per_tok, r = i % per_tok, h = r / groups, g = r % groups * VEC;
      T* o = dest(t, h);
      if (!o) continue;
      const T* src = x + (t0 + t) * p.ld_in + (long long)h * p.head_dim + d0 + g;
      float a[VEC], b[VEC];
      V::load(src, a);
      V::load(src + half, b);
      const float2* w = table + t * n + g;
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const float2 c = w[j];
        const float lo = a[j] * c.x - b[j] * c.y, hi = b[j] * c.x + a[j] * c.y;
        a[j] = lo;
        b[j] = hi;
      }
      V::store(o + d0 + g, a);
      V::store(o + d0 + g + half, b);
    }
  }
  if (waits) wait();
  // What passes through: the dimensions beyond rotary_dim of heads that move, and the values.
  const int first = cache ? p.heads : 0, tail = p.head_dim - p.rotary_dim;
  const bool moves = cache || x != out;
  if (moves && tail > 0 && turned > first) {
    const int groups = tail / VEC, per_tok = (turned - first) * groups;
    for (int i = threadIdx.x; i < nt * per_tok; i += kRopeThreads) {
      const int t = i / per_tok, r = i % per_tok, h = first + r / groups, g = p.rotary_dim + r % groups * VEC;
      T* o = dest(t, h);
      if (!o) continue;
      float a[VEC];
      V::load(x + (t0 + t) * p.ld_in + (long long)h * p.head_dim + g, a);
      V::store(o + g, a);
    }
  }
  if (cache) {
    const int groups = p.head_dim / VEC, per_tok = kv * groups;
    for (int i = threadIdx.x; i < nt * per_tok; i += kRopeThreads) {
      const int t = i / per_tok, r = i % per_tok, h = turned + r / groups, g = r % groups * VEC;
      T* o = dest(t, h);
      if (!o) continue;
      float a[VEC];
      V::load(x + (t0 + t) * p.ld_in + (long long)h * p.head_dim + g, a);
      V::store(o + g, a);
    }
  }
}

template <typename T, int VEC>
static int launch_rope(RopeParams p, cudaStream_t st) {
  // 16-byte groups when every address and both halves of a head are whole groups of them.
  auto whole = [](const void* q, long long ld) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0 && ld % VEC == 0; };
  const bool vec = whole(p.x, p.ld_in) && whole(p.out, p.ld_out) && p.head_dim % VEC == 0 && (p.rotary_dim / 2) % VEC == 0 &&
                   (!p.kc || (whole(p.kc, p.ldkv) && whole(p.vc, p.kv_batch_stride)));
  // At least four blocks an SM before a block takes several tokens.
  const long long per = p.tokens / (4LL * sm_count());
  p.tokens_per_block = (int)(per < 1 ? 1 : per > kRopeTokens ? kRopeTokens : per);
  const long long blocks = (p.tokens + p.tokens_per_block - 1) / p.tokens_per_block;
  if (blocks > 0x7fffffffLL) return kErrBadShape;
  const dim3 grid((unsigned)blocks), block(kRopeThreads);
  if (!p.kc) {
    if (vec) rope_kernel<T, VEC><<<grid, block, 0, st>>>(p);
    else     rope_kernel<T, 1><<<grid, block, 0, st>>>(p);
    return (int)cudaGetLastError();
  }
  return (int)(vec ? launch_k(rope_kernel<T, VEC>, grid, block, 0, st, p) : launch_k(rope_kernel<T, 1>, grid, block, 0, st, p));
}

}  // namespace dptb

using namespace dptb;

extern "C" int dptb_rope(const void* x, void* out, long long tokens, int heads, int head_dim, int rotary_dim,
                         int seq_len, int pos_start, float base, int inverse, int dtype, long long ld_in,
                         long long ld_out, const long long* positions, void* stream) {
  if (tokens <= 0 || heads <= 0) return 0;
  if (rotary_dim < 0 || rotary_dim % 2 || rotary_dim > head_dim) return kErrBadShape;
  RopeParams p = {};
  p.x = x; p.out = out; p.tokens = tokens; p.ld_in = ld_in; p.ld_out = ld_out;
  p.heads = heads; p.head_dim = head_dim; p.rotary_dim = rotary_dim; p.seq_len = seq_len; p.pos_start = pos_start;
  p.inverse = inverse; p.base = base; p.positions = positions;
  auto st = static_cast<cudaStream_t>(stream);
  return counted(1, dtype ? launch_rope<__nv_bfloat16, 8>(p, st) : launch_rope<float, 4>(p, st));
}

// Rows of `qkv` are [Hq | Hkv | Hkv] heads, B sequences of S rows.  Queries and keys are turned at positions
// pos0 .. pos0 + S (rotary_dim 0: not at all), keys and values go to rows row0 .. row0 + S of the caches.  With `pos_ptr`
// both starts come from the device.
extern "C" int dptb_rope_kv_append(void* qkv, long long ld, void* kc, void* vc, long long ldkv,
                                   long long kv_batch_stride, int B, int S, int Hq, int Hkv, int head_dim, int pos0,
                                   int row0, int rotary_dim, float base, int cap, const int* pos_ptr, int dtype,
                                   void* stream) {
  if (B <= 0 || S <= 0) return 0;
  if (rotary_dim < 0 || rotary_dim > head_dim || (rotary_dim & 1) || pos0 < 0 || row0 < 0 || !kc || !vc ||
      (!pos_ptr && row0 + S > cap))
    return kErrBadShape;
  RopeParams p = {};
  p.x = qkv; p.out = qkv; p.tokens = (long long)B * S; p.ld_in = ld; p.ld_out = ld;
  p.heads = Hq; p.head_dim = head_dim; p.rotary_dim = rotary_dim; p.seq_len = S; p.pos_start = pos0; p.base = base;
  p.kc = kc; p.vc = vc; p.ldkv = ldkv; p.kv_batch_stride = kv_batch_stride; p.kv_heads = Hkv; p.row0 = row0; p.cap = cap;
  p.pos_ptr = pos_ptr;
  auto st = static_cast<cudaStream_t>(stream);
  return counted(1, dtype ? launch_rope<__nv_bfloat16, 8>(p, st) : launch_rope<float, 4>(p, st));
}
