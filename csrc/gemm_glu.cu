// Gated products: out = silu(x Wg^T) * (x Wu^T), W = [gates; values] stored one below the other, in one pass of the CTA-pair GEMM.
// Without it the 2F columns leave as bf16, come back for a kernel that gates them and leave once more: 59 us beside a product of
// 255 us at 8192 x 2048 -> 2 x 5504.
#include "gemm_tc.cuh"

using namespace dptb;

// A [M, K], B [2N, K] (gates, then values), C [M, N], all bf16, no bias; M above one row tile.  kErrUnsupported for what it does not take.
extern "C" int dptb_gemm_swiglu(const DptbGemmArgs* a, void* stream) {
  if (a->M <= 0 || a->N <= 0) return 0;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (a->trans_a || !a->trans_b || a->a_f32 || a->b_f32 || a->out_f32 || a->bias || a->residual || a->aux_in || a->aux_out || a->act ||
      a->accumulate || a->alpha != 1.0f || a->K <= 0 || a->M <= kBM || a->N % 8 || a->lda % 8 || a->ldb % 8 || a->ldc % 8 || !al16(a->A) ||
      !al16(a->B) || !al16(a->C))
    return kErrUnsupported;
  GemmParams p = {};
  p.M = a->M; p.N = a->N; p.K = a->K;
  p.C = a->C; p.ldc = a->ldc;
  p.alpha = 1.0f;
  p.vec_ok = 1;
  p.tiles_m = (a->M + kBM - 1) / kBM;
  p.tiles_n = (a->N + 127) / 128;
  p.num_kb = p.kb_per_split = (a->K + kBK - 1) / kBK;
  p.splits = 1;
  const int sched = (p.tiles_m + 1) / 2;
  order_tiles(p, sched, 2ll * kBM * a->K * 2, 2ll * a->N * a->K * 2, true);
  CUtensorMap tmA, tmB;
  EpiMaps em;
  int rc = encode_tmap_2d_bf16(&tmA, a->A, (uint64_t)a->K, (uint64_t)a->M, (uint64_t)a->lda * 2, 64, kBM);
  if (!rc) rc = encode_tmap_2d_bf16(&tmB, a->B, (uint64_t)a->K, 2 * (uint64_t)a->N, (uint64_t)a->ldb * 2, 64, 128);
  if (!rc) rc = encode_tmap_2d_bf16(&em.c, a->C, (uint64_t)a->N, (uint64_t)a->M, (uint64_t)a->ldc * 2, 64, 32);
  if (rc) return rc;
  em.aux = em.in = em.c;
  return launch_tc_pair<false, false, 256, kPairStages256, true>(tmA, tmB, em, p, static_cast<cudaStream_t>(stream));
}
