"""Device attention: autograd wrappers over the tcgen05 flash-attention kernels (``csrc/attention_*.cu``).

Tensors are token-major: element ``(b, s, head, d)`` of Q lives at row ``b*S + s``, column ``head*hd + d`` of a 2-D
matrix, which is exactly what a fused QKV projection writes and what the output projection reads, so no
split / permute / concat kernels run around the attention kernel (the reference concatenates per-head results on the
host: lib/core/nn/attention/multi_head_attention.dart:167-196).
"""
from __future__ import annotations

import ctypes
import math
import os
from typing import Optional

import torch

from .. import _native as N
from . import reference as ref

c_void_p, c_int, c_ll, c_float = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float


class AttnFwdArgs(ctypes.Structure):
    _fields_ = [("q", c_void_p), ("k", c_void_p), ("v", c_void_p), ("o", c_void_p), ("lse", c_void_p),
                ("ldq", c_ll), ("ldk", c_ll), ("ldv", c_ll), ("ldo", c_ll),
                ("B", c_int), ("Sq", c_int), ("Sk", c_int), ("Hq", c_int), ("Hkv", c_int), ("head_dim", c_int),
                ("causal", c_int), ("q_offset", c_int), ("scale", c_float), ("kv_batch_rows", c_ll), ("precise", c_int)]


class AttnBwdArgs(ctypes.Structure):
    _fields_ = [("q", c_void_p), ("k", c_void_p), ("v", c_void_p), ("o", c_void_p), ("do", c_void_p),
                ("lse", c_void_p), ("delta", c_void_p), ("dq_acc", c_void_p), ("dq", c_void_p), ("dk", c_void_p),
                ("dv", c_void_p),
                ("ldq", c_ll), ("ldk", c_ll), ("ldv", c_ll), ("ldo", c_ll), ("lddo", c_ll), ("lddq", c_ll),
                ("lddk", c_ll), ("lddv", c_ll),
                ("B", c_int), ("Sq", c_int), ("Sk", c_int), ("Hq", c_int), ("Hkv", c_int), ("head_dim", c_int),
                ("causal", c_int), ("q_offset", c_int), ("scale", c_float)]


def kernel_head_dim(hd: int, backward: bool = False) -> Optional[int]:
    """Head size the tensor-core kernels run a head of ``hd`` features at: 64 and 128 directly (the backward kernel
    exists for 64 only), smaller sizes that are a multiple of 8 zero-padded to 64 (zeros add nothing to the scores and
    give zero output columns), sizes between 64 and 128 padded to 128 in forward.  ``None`` = no kernel for it."""
    if hd <= 0 or hd % 8:
        return None
    if backward and deterministic():
        return None          # the backward kernel sums dQ with fp32 atomics: run-to-run order is not fixed
    if hd <= 64:
        return 64
    if hd <= 128 and not backward:
        return 128
    return None


def deterministic() -> bool:
    """``DPTB200_DETERMINISTIC=1``: bit-identical results from run to run.  Every reduction in this package is ordered
    (two-stage column sums, split-K folded in split order, sorted embedding scatter, fixed rank order in the collective
    kernels) except the flash attention backward, whose dQ tiles from different key tiles meet in fp32 ``red.add``; with
    the flag, attention that needs gradients takes the composed GEMM + softmax path instead."""
    return os.environ.get("DPTB200_DETERMINISTIC", "0") not in ("0", "", "false", "False")


def supported_head_dim(hd: int, backward: bool = False) -> bool:
    return kernel_head_dim(hd, backward) is not None


def _wants_grad(*tensors) -> bool:
    return torch.is_grad_enabled() and any(t.requires_grad for t in tensors)


def _reads_rows(*tensors) -> bool:
    """Rows in whole 16-byte pieces: what the tensor maps describe."""
    return all(t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 for t in tensors)


def _raw_call() -> bool:
    """Whether a kernel call stands for an autograd function without gradients: no forward-mode derivatives, no transforms."""
    return torch.autograd.forward_ad._current_level < 0 and not torch._C._are_functorch_transforms_active()


def _pad_heads(x2: torch.Tensor, heads: int, hd: int, to: int) -> torch.Tensor:
    """Token-major ``[rows, heads*hd]`` -> ``[rows, heads*to]`` with zeros behind every head's features."""
    return torch.nn.functional.pad(x2.reshape(x2.shape[0], heads, hd), (0, to - hd)).reshape(x2.shape[0], heads * to)


def _to_bhsd(x2: torch.Tensor, batch: int, seq: int, heads: int, hd: int) -> torch.Tensor:
    return x2.reshape(batch, seq, heads, hd).transpose(1, 2)


def _ld(t: torch.Tensor) -> int:
    if t.dim() != 2 or t.stride(1) != 1:
        raise ValueError("attention operands must be 2-D with a contiguous last axis")
    return t.stride(0)


def attn_fwd(q2, k2, v2, B, Sq, Sk, Hq, Hkv, hd, causal, q_offset=0, scale=None, need_lse=True, out=None,
             kv_batch_rows=0, precise=False):
    """Forward kernel call on token-major 2-D views (``q2``: ``[B*Sq, >= Hq*hd]`` etc.).  Returns ``(o, lse)``.
    ``precise`` keeps the softmax weights in two bf16 parts (16 mantissa bits) for the product with V."""
    lib = N.load()
    if out is None:
        out = torch.empty(B * Sq, Hq * hd, dtype=torch.bfloat16, device=q2.device)
    lse = torch.empty(B, Hq, Sq, dtype=torch.float32, device=q2.device) if need_lse else None
    a = AttnFwdArgs()
    a.q, a.k, a.v, a.o, a.lse = q2.data_ptr(), k2.data_ptr(), v2.data_ptr(), out.data_ptr(), N.ptr(lse)
    a.ldq, a.ldk, a.ldv, a.ldo = _ld(q2), _ld(k2), _ld(v2), _ld(out)
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.head_dim = B, Sq, Sk, Hq, Hkv, hd
    a.causal, a.q_offset = int(causal), int(q_offset)
    a.scale = (1.0 / math.sqrt(hd)) if scale is None else scale
    a.kv_batch_rows = kv_batch_rows
    a.precise = int(precise)
    N.check(lib.dptb_attn_fwd(ctypes.byref(a), N.stream_ptr()), "attn_fwd")
    return out, lse


def attn_bwd(q2, k2, v2, o2, do2, lse, dq2, dk2, dv2, B, Sq, Sk, Hq, Hkv, hd, causal, q_offset=0, scale=None):
    """Backward kernel call; writes dQ / dK / dV into the given token-major 2-D views."""
    lib = N.load()
    delta = torch.empty(B, Hq, Sq, dtype=torch.float32, device=q2.device)
    dq_acc = torch.zeros(B * Sq, Hq * hd, dtype=torch.float32, device=q2.device)
    a = AttnBwdArgs()
    a.q, a.k, a.v, a.o, a.do = q2.data_ptr(), k2.data_ptr(), v2.data_ptr(), o2.data_ptr(), do2.data_ptr()
    a.lse, a.delta, a.dq_acc = lse.data_ptr(), delta.data_ptr(), dq_acc.data_ptr()
    a.dq, a.dk, a.dv = dq2.data_ptr(), dk2.data_ptr(), dv2.data_ptr()
    a.ldq, a.ldk, a.ldv, a.ldo, a.lddo = _ld(q2), _ld(k2), _ld(v2), _ld(o2), _ld(do2)
    a.lddq, a.lddk, a.lddv = _ld(dq2), _ld(dk2), _ld(dv2)
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.head_dim = B, Sq, Sk, Hq, Hkv, hd
    a.causal, a.q_offset = int(causal), int(q_offset)
    a.scale = (1.0 / math.sqrt(hd)) if scale is None else scale
    N.check(lib.dptb_attn_bwd(ctypes.byref(a), N.stream_ptr()), "attn_bwd")


class PackedAttentionFn(torch.autograd.Function):
    """Attention over a fused projection output ``qkv`` ``[B*S, (H + 2 Hkv) hd]`` -> ``[B*S, H hd]``."""

    @staticmethod
    def forward(ctx, qkv, B, S, H, Hkv, hd, causal):
        dq, dkv = H * hd, Hkv * hd
        q2, k2, v2 = qkv[:, :dq], qkv[:, dq:dq + dkv], qkv[:, dq + dkv:]
        o, lse = attn_fwd(q2, k2, v2, B, S, S, H, Hkv, hd, causal, need_lse=True)
        ctx.save_for_backward(qkv, o, lse)
        ctx.cfg = (B, S, H, Hkv, hd, causal)
        return o

    @staticmethod
    def backward(ctx, do):
        qkv, o, lse = ctx.saved_tensors
        B, S, H, Hkv, hd, causal = ctx.cfg
        dq, dkv = H * hd, Hkv * hd
        do = do if do.is_contiguous() else do.contiguous()
        dqkv = torch.empty_like(qkv)
        attn_bwd(qkv[:, :dq], qkv[:, dq:dq + dkv], qkv[:, dq + dkv:], o, do, lse,
                 dqkv[:, :dq], dqkv[:, dq:dq + dkv], dqkv[:, dq + dkv:], B, S, S, H, Hkv, hd, causal)
        return dqkv, None, None, None, None, None, None


class SeparateAttentionFn(torch.autograd.Function):
    """Attention over separate token-major ``q [B*Sq, H hd]``, ``k``/``v`` ``[B*Sk, Hkv hd]``."""

    @staticmethod
    def forward(ctx, q2, k2, v2, B, Sq, Sk, H, Hkv, hd, causal, q_offset, scale=None):
        o, lse = attn_fwd(q2, k2, v2, B, Sq, Sk, H, Hkv, hd, causal, q_offset=q_offset, scale=scale, need_lse=True)
        ctx.save_for_backward(q2, k2, v2, o, lse)
        ctx.cfg = (B, Sq, Sk, H, Hkv, hd, causal, q_offset, scale)
        return o

    @staticmethod
    def backward(ctx, do):
        q2, k2, v2, o, lse = ctx.saved_tensors
        B, Sq, Sk, H, Hkv, hd, causal, q_offset, scale = ctx.cfg
        do = do if do.is_contiguous() else do.contiguous()
        dq, dk, dv = torch.empty_like(q2), torch.empty_like(k2), torch.empty_like(v2)
        attn_bwd(q2, k2, v2, o, do, lse, dq, dk, dv, B, Sq, Sk, H, Hkv, hd, causal, q_offset=q_offset, scale=scale)
        return dq, dk, dv, None, None, None, None, None, None, None, None, None


def attn_decode_rows(q2, k3, v3, B, Sk, H, Hkv, hd):
    """One query row per sequence over all ``Sk`` rows of ``k3`` / ``v3 [B, Sk, Hkv hd]`` (cache views), no gradients."""
    from . import decode
    from .kernels import splitk_workspace
    return decode.attn_decode(q2, k3, v3, B, 1, Sk, H, Hkv, hd, Sk - 1, counters=splitk_workspace(q2.device)[1])


# ------------------------------------------------------------------------------------------------------------ fp32
class F32View(ctypes.Structure):
    _fields_ = [("p", c_void_p), ("sb", c_ll), ("ss", c_ll), ("sh", c_ll)]


class AttnF32Args(ctypes.Structure):
    _fields_ = [(n, F32View) for n in ("q", "k", "v", "o", "do", "dq", "dk", "dv")] + \
        [("lse", c_void_p), ("delta", c_void_p)] + \
        [(n, c_int) for n in ("B", "Sq", "Sk", "Hq", "Hkv", "hd", "causal", "q_offset")] + \
        [("scale", c_float), ("backward", c_int)]


def _f32_covers(B, Sq, Sk, H, Hkv, hd, q_offset=0) -> bool:
    """What ``csrc/attention_f32.cu`` takes; the composed path takes the rest."""
    return 0 < hd <= 128 and B > 0 and Sq > 0 and Sk > 0 and Hkv > 0 and H % Hkv == 0 and q_offset >= 0 and \
        max(B, H) <= 65535


def _f32_rows(t):
    return t if t.stride(-1) == 1 or t.shape[-1] == 1 else t.contiguous()


def attn_f32(q4, k4, v4, o4, causal, q_offset, lse=None, grads=None):
    """Kernel call on ``[B, S, H, hd]`` views with a contiguous last axis.  Without ``grads`` it writes ``o4`` (and ``lse
    [B, H, Sq]`` if given); with ``grads = (do, dq, dk, dv)``, views like the operands, it writes the last three."""
    B, Sq, H, hd = q4.shape
    a = AttnF32Args()
    views = (q4, k4, v4, o4) + (grads or ())
    for name, t in zip(("q", "k", "v", "o", "do", "dq", "dk", "dv"), views):
        sb, ss, sh, _ = t.stride()
        setattr(a, name, F32View(t.data_ptr(), sb, ss, sh))
    delta = torch.empty_like(lse) if grads else None
    a.lse, a.delta = N.ptr(lse), N.ptr(delta)
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.hd = B, Sq, k4.shape[1], H, k4.shape[2], hd
    a.causal, a.q_offset, a.scale, a.backward = int(causal), int(q_offset), 1.0 / math.sqrt(hd), int(grads is not None)
    N.check(N.load().dptb_attn_f32(ctypes.byref(a), N.stream_ptr()), "attn_f32")


def _f32_packed_views(x, cfg):
    B, S, H, Hkv, hd = cfg
    x4 = x.view(B, S, H + 2 * Hkv, hd)
    return x4[:, :, :H], x4[:, :, H:H + Hkv], x4[:, :, H + Hkv:]


class PackedAttentionF32Fn(torch.autograd.Function):
    """fp32 ``PackedAttentionFn``."""

    @staticmethod
    def forward(ctx, qkv, B, S, H, Hkv, hd, causal):
        qkv = qkv.contiguous()
        o = torch.empty(B * S, H * hd, dtype=qkv.dtype, device=qkv.device)
        lse = torch.empty(B, H, S, dtype=torch.float32, device=qkv.device)
        cfg = (B, S, H, Hkv, hd)
        attn_f32(*_f32_packed_views(qkv, cfg), o.view(B, S, H, hd), causal, 0, lse=lse)
        ctx.save_for_backward(qkv, o, lse)
        ctx.cfg, ctx.causal = cfg, causal
        return o

    @staticmethod
    def backward(ctx, do):
        qkv, o, lse = ctx.saved_tensors
        B, S, H, Hkv, hd = ctx.cfg
        dqkv = torch.empty_like(qkv)
        attn_f32(*_f32_packed_views(qkv, ctx.cfg), o.view(B, S, H, hd), ctx.causal, 0, lse=lse,
                 grads=(do.contiguous().view(B, S, H, hd), *_f32_packed_views(dqkv, ctx.cfg)))
        return dqkv, None, None, None, None, None, None


class AttentionF32Fn(torch.autograd.Function):
    """fp32 attention of ``[B, S, H, hd]`` views; the output is contiguous in that order."""

    @staticmethod
    def forward(ctx, q4, k4, v4, causal, q_offset):
        q4, k4, v4 = _f32_rows(q4), _f32_rows(k4), _f32_rows(v4)
        B, Sq, H, hd = q4.shape
        o = torch.empty(B, Sq, H, hd, dtype=q4.dtype, device=q4.device)
        lse = torch.empty(B, H, Sq, dtype=torch.float32, device=q4.device)
        attn_f32(q4, k4, v4, o, causal, q_offset, lse=lse)
        ctx.save_for_backward(q4, k4, v4, o, lse)
        ctx.cfg = (causal, q_offset)
        return o

    @staticmethod
    def backward(ctx, do):
        q4, k4, v4, o, lse = ctx.saved_tensors
        grads = [torch.empty(t.shape, dtype=t.dtype, device=t.device) for t in (q4, k4, v4)]
        attn_f32(q4, k4, v4, o, *ctx.cfg, lse=lse, grads=(_f32_rows(do), *grads))
        return (*grads, None, None)


def _attention_f32(q4, k4, v4, causal, q_offset):
    if _wants_grad(q4, k4, v4) or not _raw_call():     # (the function refuses derivatives and transforms that it does not have)
        return AttentionF32Fn.apply(q4, k4, v4, causal, q_offset)
    o = torch.empty(q4.shape, dtype=q4.dtype, device=q4.device)
    attn_f32(_f32_rows(q4), _f32_rows(k4), _f32_rows(v4), o, causal, q_offset)
    return o


def attention_packed(qkv, batch, seq, heads, kv_heads, head_dim, causal=True):
    """Attention over a fused projection output ``[B*S, (H + 2 Hkv) hd]`` -> ``[B*S, H hd]``."""
    d_q, d_kv = heads * head_dim, kv_heads * head_dim
    if qkv.dtype == torch.float32 and _wants_grad(qkv) and _f32_covers(batch, seq, seq, heads, kv_heads, head_dim):
        return PackedAttentionF32Fn.apply(qkv, batch, seq, heads, kv_heads, head_dim, causal)
    hd_k = kernel_head_dim(head_dim, backward=_wants_grad(qkv)) if qkv.dtype == torch.bfloat16 else None
    if hd_k == head_dim:
        return PackedAttentionFn.apply(qkv, batch, seq, heads, kv_heads, head_dim, causal)
    return attention_tokens(qkv[:, :d_q], qkv[:, d_q:d_q + d_kv], qkv[:, d_q + d_kv:], batch, seq, seq, heads, kv_heads,
                            head_dim, causal)


def attention_tokens(q2, k2, v2, batch, sq, sk, heads, kv_heads, head_dim, causal=True, q_offset=0):
    """Token-major separate operands ``q2 [B*Sq, H hd]``, ``k2`` / ``v2`` ``[B*Sk, Hkv hd]`` (with a KV cache: cache
    views) -> ``[B*Sq, H hd]``.  bf16 heads of 64 / 128 features run the tensor-core kernels as they are, other sizes as
    they are without gradients and zero-padded to the next of the two with them; what the kernels do not cover (see ``kernel_head_dim``) runs the composed path."""
    hd_k = kernel_head_dim(head_dim, backward=_wants_grad(q2, k2, v2)) if q2.dtype == torch.bfloat16 else None
    if q2.dtype == torch.float32:
        o = attention_bhsd(_to_bhsd(q2, batch, sq, heads, head_dim), _to_bhsd(k2, batch, sk, kv_heads, head_dim),
                           _to_bhsd(v2, batch, sk, kv_heads, head_dim), causal, None, q_offset)
        return o.transpose(1, 2).reshape(batch * sq, heads * head_dim)
    if hd_k is None:
        o = _attention_composed(_to_bhsd(q2, batch, sq, heads, head_dim), _to_bhsd(k2, batch, sk, kv_heads, head_dim),
                                _to_bhsd(v2, batch, sk, kv_heads, head_dim), causal, None, q_offset)
        return o.transpose(1, 2).reshape(batch * sq, heads * head_dim)
    if hd_k == head_dim:
        return SeparateAttentionFn.apply(q2, k2, v2, batch, sq, sk, heads, kv_heads, head_dim, causal, q_offset)
    if q2.shape == (batch * sq, heads * head_dim) and k2.shape == v2.shape == (batch * sk, kv_heads * head_dim) and \
            not _wants_grad(q2, k2, v2) and _reads_rows(q2, k2, v2) and _raw_call():
        # the forward kernel reads such heads as they are; only the backward one wants padded operands
        return attn_fwd(q2, k2, v2, batch, sq, sk, heads, kv_heads, head_dim, causal, q_offset=q_offset, need_lse=False)[0]
    o = SeparateAttentionFn.apply(_pad_heads(q2, heads, head_dim, hd_k), _pad_heads(k2, kv_heads, head_dim, hd_k),
                                  _pad_heads(v2, kv_heads, head_dim, hd_k), batch, sq, sk, heads, kv_heads, hd_k, causal,
                                  q_offset, 1.0 / math.sqrt(head_dim))
    return o.reshape(batch * sq, heads, hd_k)[:, :, :head_dim].reshape(batch * sq, heads * head_dim)


def attention_bhsd(q, k, v, causal=False, mask=None, q_offset=0):
    """``[B, H, S, hd]`` operands.  bf16 with a supported head size runs the tensor-core kernel (after a
    token-major relayout), fp32 without a mask the fp32 kernels on the operands as they are; anything else (odd head
    sizes, an additive mask) runs the composed device path: score GEMMs, row softmax kernel."""
    B, H, Sq, hd = q.shape
    Hkv, Sk = k.shape[1], k.shape[2]
    if q.dtype == torch.float32 and mask is None:
        # keys and values of the queries' batch, head size and device; others (values of a size of their own among them) are
        # computed, or refused, by the composed path
        if _f32_covers(B, Sq, Sk, H, Hkv, hd, q_offset) and k.shape == v.shape == (B, Hkv, Sk, hd) and \
                all(t.device == q.device and t.dtype in (torch.float32, torch.bfloat16) for t in (k, v)):
            q4, k4, v4 = (t.to(q.dtype).transpose(1, 2) for t in (q, k, v))
            return _attention_f32(q4, k4, v4, causal, q_offset).transpose(1, 2)
    if q.dtype == torch.bfloat16 and mask is None and supported_head_dim(hd, backward=_wants_grad(q, k, v)):
        q2 = q.transpose(1, 2).reshape(B * Sq, H * hd)
        k2 = k.transpose(1, 2).reshape(B * Sk, Hkv * hd)
        v2 = v.transpose(1, 2).reshape(B * Sk, Hkv * hd)
        o = attention_tokens(q2, k2, v2, B, Sq, Sk, H, Hkv, hd, causal, q_offset)
        return o.reshape(B, Sq, H, hd).transpose(1, 2)
    return _attention_composed(q, k, v, causal, mask, q_offset)


def _attention_composed(q, k, v, causal, mask, q_offset):
    """Generic path built from the library's own GEMM / softmax ops, one (batch, head) at a time."""
    from . import matmul, softmax, transpose
    from . import cuda as C
    B, H, Sq, hd = q.shape
    Hkv, Sk = k.shape[1], k.shape[2]
    g = H // Hkv
    scale = 1.0 / math.sqrt(hd)
    add = None
    if causal:
        i = torch.arange(Sq, device=q.device).unsqueeze(1) + q_offset
        j = torch.arange(Sk, device=q.device).unsqueeze(0)
        add = torch.where(j > i, -1e9, 0.0).to(q.dtype)
    if mask is not None:
        add = mask.to(q.dtype) if add is None else add + mask.to(q.dtype)
    outs = []
    for b in range(B):
        heads = []
        for h in range(H):
            qh, kh, vh = q[b, h].contiguous(), k[b, h // g].contiguous(), v[b, h // g].contiguous()
            s = C.UnaryFn.apply(matmul(qh, transpose(kh)), "scale", scale)
            if add is not None:
                s = C.BinaryFn.apply(s, add.expand(Sq, Sk).contiguous(), "add")
            heads.append(matmul(softmax(s), vh))
        outs.append(torch.stack(heads, 0))
    return torch.stack(outs, 0)
