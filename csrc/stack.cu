// A whole stack of transformer layers without gradients, launched from one native call: the kernels that the layer-by-layer
// path runs, in its order and with its arguments, without the host work of an autograd function, output allocations and
// argument blocks per kernel (about 40 to 60 us each in Python: more than most of these kernels take for a few tokens).
//
// Covers pre-norm blocks (LayerNorm or RMSNorm; two-matrix feed-forward with an activation, or gated) and post-norm blocks,
// an optional token embedding in front and an optional final norm, attention over the step's own tokens or over a
// key / value cache that the step is appended to.  Everything else is declined by the caller.
#include <math.h>
#include <string.h>

#include "common/attn_args.h"
#include "common/gemm_args.h"
#include "common/host.h"

using namespace dptb;

extern "C" {
int dptb_gemm(const DptbGemmArgs*, void*);
int dptb_gemm_skinny(const DptbGemmArgs*, const DptbTpArArgs*, void*);
int dptb_gemm_swiglu(const DptbGemmArgs*, void*);
int dptb_gemm_skinny_swiglu(const DptbGemmArgs*, void*);
int dptb_attn_f32_append(const DptbAttnF32Args*, const DptbF32View*, const DptbF32View*, void*);
int dptb_attn_fwd(const DptbAttnFwdArgs*, void*);
int dptb_attn_f32(const DptbAttnF32Args*, void*);
int dptb_attn_decode(const DptbDecodeArgs*, void*);
int dptb_attn_decode_splits_hd(int, int, int, int, int);
long long dptb_attn_decode_ws_floats(int, int, int, int, int);
int dptb_rope_kv_append(void*, long long, void*, void*, long long, long long, int, int, int, int, int, int, int, int, float, int,
                        const int*, int, void*);
int dptb_rope(const void*, void*, long long, int, int, int, int, int, float, int, int, long long, long long, const long long*, void*);
int dptb_layernorm_fwd(const void*, const void*, const void*, void*, float*, float*, long long, int, float, int, void*);
int dptb_rmsnorm_fwd(const void*, const void*, void*, float*, long long, int, float, int, void*);
int dptb_swiglu_fwd(const void*, long long, const void*, long long, void*, long long, long long, int, int, void*);
int dptb_binary(const void*, const void*, void*, long long, long long, int, int, int, void*);
int dptb_embedding_fwd(const void*, long long, const long long*, const void*, long long, int, int, void*, long long, int, int, void*);
}

// Pointers of one layer, in this order in the table that the caller passes.
enum StackSlot { kN1G, kN1B, kQkvW, kQkvB, kWoW, kWoB, kN2G, kN2B, kUpW, kUpB, kDownW, kDownB, kKCache, kVCache, kStackSlots };

struct DptbStackArgs {
  int layers, bf16, post_norm, rms, gated, act;       // act: the forward codes of dptb_gemm
  int B, S, D, H, Hkv, hd, F;
  int causal, start_pos, rotary_dim;
  int cached, past, cap;                              // cached: rows `past`.. of the caches receive the step
  int skinny_rows;                                    // rows up to which bf16 x W^T streams the weight (0: never)
  int num_counters;
  float eps, rope_base, final_eps, embed_eps;
  long long ldkv, kv_batch_stride;
  const void* x;                                      // [B * S, D], or null: tokens
  void* out;                                          // [B * S, D]
  const void* final_g;
  const void* final_b;
  // embedding: table rows (+ position rows) (+ one row added everywhere) (, LayerNorm)
  const long long* tokens;
  const void* table;
  const void* pos_table;
  const void* add_row;
  const void* embed_g;
  const void* embed_b;
  long long vocab, pos_rows;
  int pos_start, reserved;
  void* ws;                                           // scratch of dptb_stack_ws_bytes bytes
  void* gemm_ws;                                      // split-K scratch and counters of the current stream
  long long gemm_ws_bytes;
  int* counters;
};

namespace {
struct Layout {
  long long norm, qkv, attn, h0, h1, h2, up, act, stats, dec, total;
  int dec_splits;
};
// The rule of the layer-by-layer path (see there): one query row per sequence over a cache.
bool split_decode(const DptbStackArgs* a) {
  return a->bf16 && a->cached && a->S == 1 && (a->hd == 64 || a->hd == 128) && a->H / a->Hkv <= 8;
}
Layout layout(const DptbStackArgs* a) {
  Layout l;
  const long long rows = (long long)a->B * a->S, esz = a->bf16 ? 2 : 4;
  long long at = 0;
  auto take = [&](long long bytes) { const long long p = at; at += (bytes + 255) / 256 * 256; return p; };
  l.norm = take(rows * a->D * esz);
  l.qkv = take(rows * (a->H + 2 * a->Hkv) * a->hd * esz);
  l.attn = take(rows * a->H * a->hd * esz);
  l.h0 = take(rows * a->D * esz);
  l.h1 = take(rows * a->D * esz);
  l.h2 = take(rows * a->D * esz);
  l.up = take(rows * a->F * (a->gated ? 2 : 1) * esz);
  l.act = a->gated ? take(rows * a->F * esz) : l.up;
  l.stats = take(rows * 8);
  l.dec_splits = split_decode(a) ? dptb_attn_decode_splits_hd(a->B, 1, a->Hkv, a->past + 1, a->hd) : 0;
  l.dec = take(l.dec_splits > 0 ? dptb_attn_decode_ws_floats(a->B, 1, a->H, a->hd, l.dec_splits) * 4 : 0);
  l.total = at;
  return l;
}
}  // namespace

extern "C" long long dptb_stack_ws_bytes(const DptbStackArgs* a) { return layout(a).total; }

static int stack_launch(const DptbStackArgs* a, const void* const* table, void* stream) {
  const long long rows = (long long)a->B * a->S;
  if (rows <= 0 || a->layers <= 0) return kErrBadShape;
  if (rows > 0x7fffffffLL || a->H <= 0 || a->Hkv <= 0 || a->H % a->Hkv) return kErrBadShape;
  const Layout l = layout(a);
  char* ws = static_cast<char*>(a->ws);
  const int M = (int)rows, D = a->D, hd = a->hd, dq = a->H * hd, dkv = a->Hkv * hd, ldqkv = dq + 2 * dkv;
  const long long esz = a->bf16 ? 2 : 4;
  float* stats = reinterpret_cast<float*>(ws + l.stats);
  const float scale = (float)(1.0 / sqrt((double)hd));

  auto norm = [&](const void* x, const void* g, const void* b, void* y, float eps, bool rms) {
    return rms ? dptb_rmsnorm_fwd(x, g, y, stats, rows, D, eps, a->bf16, stream)
               : dptb_layernorm_fwd(x, g, b, y, stats, stats + rows, rows, D, eps, a->bf16, stream);
  };
  auto linear = [&](const void* x, int K, const void* w, const void* bias, int N, void* y, int act, const void* residual) {
    DptbGemmArgs g;
    memset(&g, 0, sizeof(g));
    g.A = x; g.B = w; g.C = y; g.bias = bias; g.residual = residual;
    g.lda = K; g.ldb = K; g.ldc = N; g.ldr = N;
    g.M = M; g.N = N; g.K = K;
    g.trans_b = 1;
    g.a_f32 = g.b_f32 = g.out_f32 = g.bias_f32 = g.epi_f32 = a->bf16 ? 0 : 1;
    g.act = act; g.alpha = 1.0f;
    g.ws = a->gemm_ws; g.ws_bytes = a->gemm_ws_bytes;
    g.counters = a->counters; g.num_counters = a->num_counters;
    if (a->bf16 && M <= a->skinny_rows) {
      const int rc = dptb_gemm_skinny(&g, nullptr, stream);
      if (rc != kErrUnsupported) return rc;
    }
    return dptb_gemm(&g, stream);
  };
  // The two products of a gated unit and the gate: one kernel where it exists, else the product of both and a pass over it.
  auto gated = [&](const void* x, const void* w, const void* bias, char* up, void* y) {
    if (a->bf16 && !bias) {
      DptbGemmArgs g;
      memset(&g, 0, sizeof(g));
      g.A = x; g.B = w; g.C = y;
      g.lda = g.ldb = D; g.ldc = a->F;
      g.M = M; g.N = a->F; g.K = D;
      g.trans_b = 1; g.alpha = 1.0f;
      const int rc = M <= a->skinny_rows ? dptb_gemm_skinny_swiglu(&g, stream) : dptb_gemm_swiglu(&g, stream);
      if (rc != kErrUnsupported) return rc;
    }
    const int rc = linear(x, D, w, bias, 2 * a->F, up, 0, nullptr);
    return rc ? rc : dptb_swiglu_fwd(up, 2LL * a->F, up + a->F * esz, 2LL * a->F, y, a->F, rows, a->F, a->bf16, stream);
  };
  auto attend = [&](char* qkv, const void* kc, const void* vc, void* o, bool append) {
    const int Sk = a->cached ? a->past + a->S : a->S;
    const char* k = a->cached ? static_cast<const char*>(kc) : qkv + dq * esz;
    const char* v = a->cached ? static_cast<const char*>(vc) : qkv + (dq + dkv) * esz;
    const long long ldk = a->cached ? a->ldkv : ldqkv;
    const long long batch = a->cached ? a->kv_batch_stride : (long long)a->S * ldqkv;
    if (!a->bf16) {
      DptbAttnF32Args f;
      memset(&f, 0, sizeof(f));
      f.q = {reinterpret_cast<float*>(qkv), (long long)a->S * ldqkv, ldqkv, hd};
      f.k = {reinterpret_cast<float*>(const_cast<char*>(k)), batch, ldk, hd};
      f.v = {reinterpret_cast<float*>(const_cast<char*>(v)), batch, ldk, hd};
      f.o = {static_cast<float*>(o), (long long)a->S * dq, dq, hd};
      f.B = a->B; f.Sq = a->S; f.Sk = Sk; f.Hq = a->H; f.Hkv = a->Hkv; f.hd = hd;
      f.causal = a->causal; f.q_offset = a->cached ? a->past : 0; f.scale = scale;
      if (!append) return dptb_attn_f32(&f, stream);
      const DptbF32View kn = {reinterpret_cast<float*>(qkv) + dq, (long long)a->S * ldqkv, ldqkv, hd};
      const DptbF32View vn = {reinterpret_cast<float*>(qkv) + dq + dkv, (long long)a->S * ldqkv, ldqkv, hd};
      return dptb_attn_f32_append(&f, &kn, &vn, stream);
    }
    if (l.dec_splits > 0) {
      DptbDecodeArgs d;
      memset(&d, 0, sizeof(d));
      d.q = qkv; d.k = k; d.v = v; d.o = o;
      d.ws = reinterpret_cast<float*>(ws + l.dec); d.ws_floats = (l.total - l.dec) / 4;
      d.ldq = ldqkv; d.ldkv = ldk; d.ldo = dq; d.kv_batch_stride = batch;
      d.B = a->B; d.Sq = 1; d.Sk = Sk; d.Hq = a->H; d.Hkv = a->Hkv; d.head_dim = hd;
      d.splits = l.dec_splits; d.q_offset = Sk - 1; d.scale = scale; d.cap = a->cap;
      d.num_counters = a->num_counters; d.counters = reinterpret_cast<unsigned int*>(a->counters);
      return dptb_attn_decode(&d, stream);
    }
    DptbAttnFwdArgs f;
    memset(&f, 0, sizeof(f));
    f.q = qkv; f.k = k; f.v = v; f.o = o;
    f.ldq = ldqkv; f.ldk = ldk; f.ldv = ldk; f.ldo = dq;
    f.B = a->B; f.Sq = a->S; f.Sk = Sk; f.Hq = a->H; f.Hkv = a->Hkv; f.head_dim = hd;
    f.causal = a->causal; f.q_offset = a->cached ? a->past : 0; f.scale = scale;
    f.kv_batch_rows = a->cached ? batch / ldk : 0;
    return dptb_attn_fwd(&f, stream);
  };

#define DPTB_STACK_OK(expr) do { const int rc_ = (expr); if (rc_) return rc_; } while (0)
  const void* cur = a->x;
  if (!cur) {
    // the last of embedding, added row and norm that there is leaves the input in h0
    void* e = a->add_row || a->embed_g ? ws + l.h1 : ws + l.h0;
    DPTB_STACK_OK(dptb_embedding_fwd(a->table, a->vocab, a->tokens, a->pos_table, a->pos_rows, a->pos_start, a->S, e, rows, D,
                                     a->bf16, stream));
    if (a->add_row) {
      void* s = a->embed_g ? ws + l.h2 : ws + l.h0;
      DPTB_STACK_OK(dptb_binary(e, a->add_row, s, rows * D, D, 0, 2, a->bf16, stream));
      e = s;
    }
    if (a->embed_g) {
      DPTB_STACK_OK(norm(e, a->embed_g, a->embed_b, ws + l.h0, a->embed_eps, false));
      e = ws + l.h0;
    }
    cur = e;
  }
  char* qkv = ws + l.qkv;
  char* mid = ws + l.h1;
  for (int i = 0; i < a->layers; ++i) {
    const void* const* t = table + (long long)i * kStackSlots;
    const bool last = i + 1 == a->layers;
    const void* x = cur;
    if (!a->post_norm) {
      DPTB_STACK_OK(norm(cur, t[kN1G], t[kN1B], ws + l.norm, a->eps, a->rms));
      x = ws + l.norm;
    }
    {
      // A product that opens the chain is launched as usual: the kernel ahead of it is not of the chain and may have written its weight.
      int& pdl = pdl_flag();
      const int chain = pdl;
      if (x == a->x) pdl = 0;
      const int rc = linear(x, D, t[kQkvW], t[kQkvB], ldqkv, qkv, 0, nullptr);
      pdl = chain;
      if (rc) return rc;
    }
    // Few fp32 rows that are not turned: the attention appends them to the caches itself.
    int attended = kErrUnsupported;
    if (a->cached && !a->bf16 && a->rotary_dim == 0 && a->past + a->S <= a->cap)
      attended = attend(qkv, t[kKCache], t[kVCache], ws + l.attn, true);
    if (attended == kErrUnsupported) {
      if (a->cached) {
        DPTB_STACK_OK(dptb_rope_kv_append(qkv, ldqkv, const_cast<void*>(t[kKCache]), const_cast<void*>(t[kVCache]), a->ldkv,
                                          a->kv_batch_stride, a->B, a->S, a->H, a->Hkv, hd, a->start_pos, a->past,
                                          a->rotary_dim, a->rope_base, a->cap, nullptr, a->bf16, stream));
      } else if (a->rotary_dim > 0) {
        DPTB_STACK_OK(dptb_rope(qkv, qkv, rows, a->H + a->Hkv, hd, a->rotary_dim, a->S, a->start_pos, a->rope_base, 0, a->bf16,
                                ldqkv, ldqkv, nullptr, stream));
      }
      attended = attend(qkv, t[kKCache], t[kVCache], ws + l.attn, false);
    }
    DPTB_STACK_OK(attended);
    DPTB_STACK_OK(linear(ws + l.attn, dq, t[kWoW], t[kWoB], D, mid, 0, cur));          // mid = attention + residual
    const void* y = ws + l.norm;
    const void* res = mid;
    if (a->post_norm) {
      DPTB_STACK_OK(norm(mid, t[kN1G], t[kN1B], ws + l.norm, a->eps, a->rms));
      res = ws + l.norm;
    } else {
      DPTB_STACK_OK(norm(mid, t[kN2G], t[kN2B], ws + l.norm, a->eps, a->rms));
    }
    const void* f = ws + l.up;
    if (a->gated) {
      DPTB_STACK_OK(gated(y, t[kUpW], t[kUpB], ws + l.up, ws + l.act));
      f = ws + l.act;
    } else {
      DPTB_STACK_OK(linear(y, D, t[kUpW], t[kUpB], a->F, ws + l.up, a->act, nullptr));
    }
    // The layer's output: the caller's buffer when nothing follows, else h2 and h0 in turn (the input is dead by now).
    char* next = cur == ws + l.h2 ? ws + l.h0 : ws + l.h2;
    if (a->post_norm) {
      DPTB_STACK_OK(linear(f, a->F, t[kDownW], t[kDownB], D, mid, 0, res));
      void* o = last ? a->out : next;
      DPTB_STACK_OK(norm(mid, t[kN2G], t[kN2B], o, a->eps, a->rms));
      cur = o;
    } else {
      void* o = last && !a->final_g ? a->out : next;
      DPTB_STACK_OK(linear(f, a->F, t[kDownW], t[kDownB], D, o, 0, res));
      cur = o;
    }
  }
  if (!a->post_norm && a->final_g) DPTB_STACK_OK(norm(cur, a->final_g, a->final_b, a->out, a->final_eps, a->rms));
#undef DPTB_STACK_OK
  return 0;
}

// The kernels of a step start as programmatic dependents of one another, so that their set-up, and the first weights of the products of few
// rows, overlap the end of the kernel before.  Which steps gain was measured as called, with and without (B200):
//   bf16   1.0 to 1.15 times as fast up to 64 rows (stacks of 3 layers, widths 128 to 2048, a prompt and one token each); beyond, products
//          and attention wait at their top: 64 x 119 tokens of width 384 693 -> 606 us, 300 tokens of width 2048 946 -> 832, 128 tokens
//          over 300 each 737 -> 607, 256 x 119 of width 384 1730 -> 1673, but 4 x 2048 of width 2048 4545 -> 4568.
//   fp32   (stacks of 4 layers) 1.05 to 1.37 times as fast at 1 to 64 rows of widths 128 to 1024, 1.18 to 1.28 at 72 to 128 rows of widths
//          up to 768; sequences of up to 128: 1.15 at 8 x 119 rows of 384, 1.07 at 509 tokens, one each, of 768.  Longer sequences: 1.18
//          at 256 rows of 384, but 0.91 at 509 of 768, where all rows have the same keys: CTAs that start where an SM is free crowd on the
//          first ones.  Causal rows, the longest first, stand that better: up to 640 rows 1.09 to 1.19 at widths 256 to 512, 1.04 at 509 and
//          512 of 768, 1.00 at 640 of 512 and 768; from 768 rows on 1.07 to 1.10 at width 256, 0.92 to 1.06 at 384, 0.96 to 1.04 at 512, 0.88
//          at 768.
constexpr long long kChainedArea = 12 << 20, kChainedAreaF32 = 384 << 10, kChainedAreaF32Rows = 256 << 10, kChainedAreaF32Long = 128 << 10;
static bool chained(const DptbStackArgs* a) {
  const long long area = (long long)a->B * a->S * a->D;
  if (a->bf16) return area <= kChainedArea;
  if (a->S <= 128) return area <= kChainedAreaF32;
  return area <= (!a->causal ? kChainedAreaF32Long : a->S <= 640 ? kChainedAreaF32 : kChainedAreaF32Rows);
}
extern "C" int dptb_stack_infer(const DptbStackArgs* a, const void* const* table, void* stream) {
  int& pdl = pdl_flag();
  const int before = pdl;
  if (chained(a)) pdl = 1;
  const int rc = stack_launch(a, table, stream);
  pdl = before;
  return rc;
}
