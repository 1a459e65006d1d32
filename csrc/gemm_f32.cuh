// Parameters and epilogue of the fp32 GEMM kernels (gemm_f32.cu: multiply-adds; gemm_f32_tc.cu: matrix instructions).
#pragma once
#include <cuda_bf16.h>

#include "common/gemm_args.h"
#include "common/host.h"
#include "common/ptx.cuh"

namespace dptb {

struct GemmF32Params {
  const float* A;
  const float* B;
  float* C;
  const void* bias;
  const float* residual;
  float* aux_out;
  const float* aux_in;
  long long lda, ldb, ldc, ldr, ld_aux_out, ld_aux_in;
  int M, N, K;
  int bias_f32, accumulate, act;
  float alpha;
  int vec_a, vec_b, vec_c;   // 16-byte accesses allowed (base and leading dimension)
  int splits, k_per_split;   // k_per_split is a multiple of kF32BK
  float* ws;
  int* counters;
};

// Activations as the elementwise kernels compute them (accurate tanh / exp): the values do not depend on whether the
// activation is fused.
__device__ __forceinline__ float act_f32(int act, float x) {
  switch (act) {
    case 1: return fmaxf(x, 0.0f);
    case 2: return 0.5f * x * (1.0f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    case 3: return x / (1.0f + expf(-1.702f * x));
    case 4: return x / (1.0f + expf(-x));
    default: return x;
  }
}
__device__ __forceinline__ float act_grad_f32(int act, float x) {
  switch (act) {
    case 11: return x > 0.0f ? 1.0f : 0.0f;
    case 12: {
      const float t = tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x));
      return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x * x);
    }
    case 13: {
      const float s = 1.0f / (1.0f + expf(-1.702f * x));
      return s + 1.702f * x * s * (1.0f - s);
    }
    case 14: {
      const float s = 1.0f / (1.0f + expf(-x));
      return s * (1.0f + x * (1.0f - s));
    }
    case 15: return x;
    default: return 1.0f;
  }
}
__device__ __forceinline__ void epilogue_f32(const GemmF32Params& p, long long row, int col, float v) {
  v *= p.alpha;
  if (p.bias) v += p.bias_f32 ? static_cast<const float*>(p.bias)[col] : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col]);
  if (p.aux_out) p.aux_out[row * p.ld_aux_out + col] = v;
  if (p.act >= 11) v *= act_grad_f32(p.act, p.aux_in[row * p.ld_aux_in + col]);
  else if (p.act) v = act_f32(p.act, v);
  if (p.residual) v += p.residual[row * p.ldr + col];
  float* c = p.C + row * p.ldc + col;
  *c = p.accumulate ? *c + v : v;
}
// Four neighbouring columns; every buffer takes 16-byte accesses (vec_c).
__device__ __forceinline__ void epilogue_f32x4(const GemmF32Params& p, long long row, int col, float4 v4) {
  float v[4] = {v4.x * p.alpha, v4.y * p.alpha, v4.z * p.alpha, v4.w * p.alpha};
  if (p.bias) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] += p.bias_f32 ? static_cast<const float*>(p.bias)[col + j]
                         : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col + j]);
  }
  if (p.aux_out) *reinterpret_cast<float4*>(p.aux_out + row * p.ld_aux_out + col) = make_float4(v[0], v[1], v[2], v[3]);
  if (p.act >= 11) {
    const float4 x = *reinterpret_cast<const float4*>(p.aux_in + row * p.ld_aux_in + col);
    v[0] *= act_grad_f32(p.act, x.x); v[1] *= act_grad_f32(p.act, x.y);
    v[2] *= act_grad_f32(p.act, x.z); v[3] *= act_grad_f32(p.act, x.w);
  } else if (p.act) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = act_f32(p.act, v[j]);
  }
  if (p.residual) {
    const float4 r = *reinterpret_cast<const float4*>(p.residual + row * p.ldr + col);
    v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
  }
  float4* c = reinterpret_cast<float4*>(p.C + row * p.ldc + col);
  if (p.accumulate) {
    const float4 o = *c;
    v[0] = o.x + v[0]; v[1] = o.y + v[1]; v[2] = o.z + v[2]; v[3] = o.w + v[3];
  }
  *c = make_float4(v[0], v[1], v[2], v[3]);
}

// Tensor-core tiles (gemm_f32_tc.cu) of bn = 64 or 128 columns, K in p.splits <= 8 non-empty parts of p.k_per_split terms (a multiple
// of 64); the choice of both, and the time that it is expected to take in microseconds.
constexpr int kF32TcBK = 64;
double f32_tc_plan(int M, int N, int K, int* bn, int* splits);
cudaError_t launch_f32_tc(const GemmF32Params& p, int bn, bool amn, bool bmn, cudaStream_t st);

}  // namespace dptb
