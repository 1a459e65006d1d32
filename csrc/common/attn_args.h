// Argument blocks of the attention entry points (mirrored by ctypes.Structure classes in Python), shared by the translation
// units that implement and call them.
#pragma once

// dptb_attn_fwd
struct DptbAttnFwdArgs {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  float* lse;
  long long ldq, ldk, ldv, ldo;
  int B, Sq, Sk, Hq, Hkv, head_dim;
  int causal, q_offset;
  float scale;
  long long kv_batch_rows;  // rows between consecutive batches of K / V (a cache's capacity); 0 = Sk
  int precise;              // softmax weights as two bf16 parts
};

// dptb_attn_decode
struct DptbDecodeArgs {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  float* ws;
  long long ws_floats;
  long long ldq, ldkv, ldo, kv_batch_stride;
  int B, Sq, Sk, Hq, Hkv, head_dim, splits, q_offset;
  float scale;
  const int* pos_ptr;
  int cap;
  int num_counters;
  unsigned int* counters;   // arrival words of this call (zero before and after it), or null: the shared table
};

// dptb_attn_f32
struct DptbF32View {
  float* p;
  long long sb, ss, sh;
};
struct DptbAttnF32Args {
  DptbF32View q, k, v, o, dout, dq, dk, dv;      // backward only: dout, dq, dk, dv
  float* lse;      // [B, Hq, Sq]; forward: written unless null, backward: read
  float* delta;    // backward scratch of the same size
  int B, Sq, Sk, Hq, Hkv, hd, causal, q_offset;
  float scale;
  int backward;
};
