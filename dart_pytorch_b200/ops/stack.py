"""Transformer stacks without gradients as one native call (``csrc/stack.cu``).

Under ``torch.no_grad()`` the layers' kernels are launched from C++, with the same arguments and in the same order as by the
modules; only the host work between them goes.  ``run`` returns ``None`` for whatever it does not cover, and the modules'
own forward passes then run (and raise their errors)."""
from __future__ import annotations

import ctypes
from typing import Optional, Sequence

import torch

from .. import _native as N
from . import kernels as K

c_void_p, c_int, c_ll, c_float = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float


class StackArgs(ctypes.Structure):
    _fields_ = [(n, c_int) for n in ("layers", "bf16", "post_norm", "rms", "gated", "act", "B", "S", "D", "H", "Hkv", "hd", "F",
                                     "causal", "start_pos", "rotary_dim", "cached", "past", "cap", "skinny_rows",
                                     "num_counters")] + \
        [(n, c_float) for n in ("eps", "rope_base", "final_eps", "embed_eps")] + \
        [(n, c_ll) for n in ("ldkv", "kv_batch_stride")] + \
        [(n, c_void_p) for n in ("x", "out", "final_g", "final_b", "tokens", "table", "pos_table", "add_row", "embed_g",
                                 "embed_b")] + \
        [("vocab", c_ll), ("pos_rows", c_ll), ("pos_start", c_int), ("reserved", c_int), ("ws", c_void_p),
         ("gemm_ws", c_void_p), ("gemm_ws_bytes", c_ll), ("counters", c_void_p)]


class Layer:
    """What ``run`` takes of one layer: the module's attention, its two norms and feed-forward parameters."""
    __slots__ = ("attn", "norm1", "norm2", "up_w", "up_b", "down_w", "down_b")

    def __init__(self, attn, norm1, norm2, up_w, up_b, down_w, down_b):
        self.attn, self.norm1, self.norm2 = attn, norm1, norm2
        self.up_w, self.up_b, self.down_w, self.down_b = up_w, up_b, down_w, down_b


def plain(module, cls) -> bool:
    """A module of exactly this class, neither of whose forward methods has been replaced on the object."""
    if type(module) is not cls:
        return False
    own = module.__dict__
    return "forward" not in own and "with_residual" not in own


def eligible(t: torch.Tensor) -> bool:
    """Whether raw kernel calls stand for the ops on ``t``: no gradients, forward-mode derivatives, transforms, tracing or
    dispatch modes, and an ordinary tensor on the current device."""
    return not torch.is_grad_enabled() and t.is_cuda and type(t) in (torch.Tensor, torch.nn.Parameter) and \
        t.device.index == torch.cuda.current_device() and not torch._C._are_functorch_transforms_active() and \
        torch._C._len_torch_dispatch_stack() == 0 and torch._C._len_torch_function_stack() == 0 and \
        torch._C._get_tracing_state() is None and torch.autograd.forward_ad._current_level < 0


_lib_ready = False


def _lib():
    """The native library, or None when it is a component build without this entry point."""
    global _lib_ready
    lib = N.load()
    if not _lib_ready:
        if getattr(lib, "dptb_stack_infer", None) is None:
            return None
        lib.dptb_stack_ws_bytes.argtypes = [ctypes.POINTER(StackArgs)]
        lib.dptb_stack_ws_bytes.restype = c_ll
        lib.dptb_stack_infer.argtypes = [ctypes.POINTER(StackArgs), c_void_p, c_void_p]
        lib.dptb_stack_infer.restype = c_int
        _lib_ready = True
    return lib


def run(layers: Sequence[Layer], x: Optional[torch.Tensor], *, post_norm=False, rms=False, gated=False, act=None, causal=False,
        start_pos: int = 0, caches=None, final_norm=None, tokens=None, table=None, pos_table=None, pos_start: int = 0,
        add_row=None, embed_norm=None) -> Optional[torch.Tensor]:
    """Hidden states after ``layers`` (and ``final_norm``) for an input ``x [N, D]`` / ``[B, N, D]``, or for ``tokens`` looked
    up in ``table`` (plus position rows, plus ``add_row``, then ``embed_norm``).  ``caches``: one ``MHACache`` per layer, to
    which the step's keys and values are appended."""
    src = x if tokens is None else tokens
    like = x if tokens is None else table
    lib = _lib() if layers and eligible(src) else None
    if lib is None or src.numel() == 0:
        return None
    src = src.contiguous()
    dtype, dev = like.dtype, src.device
    lead = src.shape[:-1] if tokens is None else src.shape
    if len(lead) not in (1, 2) or dtype not in (torch.bfloat16, torch.float32):
        return None
    at = layers[0].attn
    D, H, Hkv, hd, rope = at.embed_dim, at.num_heads, at.num_kv_heads, at.head_dim, at.rope
    F = layers[0].down_w.shape[-1]
    B, S = (lead[0] if len(lead) == 2 else 1), lead[-1]
    bf16 = dtype == torch.bfloat16
    if tokens is None and x.shape[-1] != D or max(B, H) > 65535:
        return None
    if bf16:
        if hd <= 0 or hd > 128 or hd % 8:
            return None
    elif hd > 128:
        return None
    if rope is not None and not 0 <= start_pos <= rope.max_ctx - S:
        return None
    if act not in (None, "relu", "gelu_tanh", "quick_gelu", "silu"):
        return None

    def ok(t, *shape):
        return t.dtype == dtype and t.device == dev and t.shape == shape and t.is_contiguous()

    def vec(t, n):
        return t is None or (t.dtype == dtype and t.device == dev and t.numel() == n and t.is_contiguous())
    nq, gamma_beta = (H + 2 * Hkv) * hd, not rms
    ptrs = []
    for lay in layers:
        a, n1, n2 = lay.attn, lay.norm1, lay.norm2
        if (a.embed_dim, a.num_heads, a.num_kv_heads, a.head_dim) != (D, H, Hkv, hd) or n1.eps != n2.eps or \
                n1.eps != layers[0].norm1.eps or a.rope is not rope and (
                    a.rope is None or rope is None or (a.rope.rotary_dim, a.rope.base, a.rope.max_ctx) !=
                    (rope.rotary_dim, rope.base, rope.max_ctx)):
            return None
        wo = a.wo
        b1, b2 = (n1.beta, n2.beta) if gamma_beta else (None, None)
        if not (ok(a.w_qkv, nq, D) and ok(wo.weight, D, H * hd) and ok(lay.up_w, 2 * F if gated else F, D) and
                ok(lay.down_w, D, F) and vec(a.b_qkv, nq) and vec(wo.bias, D) and vec(lay.up_b, F) and vec(lay.down_b, D) and
                vec(n1.gamma, D) and vec(b1, D) and vec(n2.gamma, D) and vec(b2, D)):
            return None
        ptrs += [N.ptr(t) for t in (n1.gamma, b1, a.w_qkv, a.b_qkv, wo.weight, wo.bias, n2.gamma, b2, lay.up_w, lay.up_b,
                                    lay.down_w, lay.down_b)] + [None, None]
    for norm in (final_norm, embed_norm):
        if norm is not None and not (vec(norm.gamma, D) and vec(getattr(norm, "beta", None), D)):
            return None
    a = StackArgs()
    if tokens is not None:
        if tokens.dtype != torch.long or not ok(table, table.shape[0], D) or not vec(add_row, D) or \
                pos_table is not None and not ok(pos_table, pos_table.shape[0], D):
            return None
        a.tokens, a.table, a.pos_table, a.add_row = src.data_ptr(), table.data_ptr(), N.ptr(pos_table), N.ptr(add_row)
        a.vocab, a.pos_rows, a.pos_start = table.shape[0], 0 if pos_table is None else pos_table.shape[0], pos_start
        if embed_norm is not None:
            a.embed_g, a.embed_b, a.embed_eps = embed_norm.gamma.data_ptr(), embed_norm.beta.data_ptr(), embed_norm.eps
    else:
        a.x = src.data_ptr()
    if caches is not None:
        past, width = caches[0].seq_len, Hkv * hd
        for c in caches:
            k, v = c.k_buf, c.v_buf
            if c.seq_len != past or k is not None and (
                    k.dtype != dtype or v.dtype != dtype or k.device != dev or v.device != dev or
                    k.shape[0] != B or k.shape[2] != width or not k.is_contiguous() or not v.is_contiguous() or
                    k.shape != v.shape or bf16 and (k.data_ptr() | v.data_ptr()) % 16):     # (bf16 rows go in 16-byte pieces)
                return None
        if len({id(c) for c in caches}) != len(caches):
            return None
        for c in caches:
            c._ensure(B, past + S, width, like)
        if any(c.k_buf.shape != caches[0].k_buf.shape for c in caches):
            return None
        for i, c in enumerate(caches):
            ptrs[14 * i + 12], ptrs[14 * i + 13] = c.k_buf.data_ptr(), c.v_buf.data_ptr()
        a.cached, a.past, a.cap = 1, past, caches[0].k_buf.shape[1]
        a.ldkv, a.kv_batch_stride = width, a.cap * width
    a.layers, a.bf16, a.post_norm, a.rms, a.gated = len(layers), int(bf16), int(post_norm), int(rms), int(gated)
    a.act = K.ACT_CODES[act]
    a.B, a.S, a.D, a.H, a.Hkv, a.hd, a.F = B, S, D, H, Hkv, hd, F
    a.causal, a.start_pos = int(causal), start_pos
    if rope is not None:
        a.rotary_dim, a.rope_base = rope.rotary_dim, rope.base
    a.eps = layers[0].norm1.eps
    if final_norm is not None:
        a.final_g, a.final_b, a.final_eps = final_norm.gamma.data_ptr(), N.ptr(getattr(final_norm, "beta", None)), final_norm.eps
    a.skinny_rows = K.SKINNY_MAX_ROWS if K._SKINNY_ON else 0
    ws, counters = K.splitk_workspace(dev)
    a.gemm_ws, a.gemm_ws_bytes, a.counters, a.num_counters = ws.data_ptr(), ws.numel(), counters.data_ptr(), counters.numel()
    scratch = torch.empty(lib.dptb_stack_ws_bytes(ctypes.byref(a)), dtype=torch.uint8, device=dev)
    out = torch.empty(*lead, D, dtype=dtype, device=dev)
    a.ws, a.out = scratch.data_ptr(), out.data_ptr()
    N.check(lib.dptb_stack_infer(ctypes.byref(a), (c_void_p * len(ptrs))(*ptrs), N.stream_ptr()), "stack_infer")
    if caches is not None:
        torch.autograd.graph.increment_version([t for c in caches for t in (c.k_buf, c.v_buf)])     # written in place
        for c in caches:
            c.seq_len += S
            c.__dict__.pop("_fills", None)
    return out
