"""bf16 GEMM with K split over CTAs that fold their tile together, in bands of row tiles, and with outputs whose width is no multiple
of 8, against fp32."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K
from dart_pytorch_b200.ops import reference as R


def _mk(shape, seed, pad=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape[0], shape[1] + pad, device="cuda", generator=g) * scale).bfloat16()[:, :shape[1]]


def _close(out, ref, *steps):
    """fp32 sums of exact products; the result, and where an epilogue is staged in bf16 what stands before each step, is rounded once
    (2^-8 of its size at most)."""
    size = ref.abs() + sum(t.abs() for t in steps)
    assert ((out.float() - ref).abs() <= 1.01 * 2.0 ** -8 * size + 1e-4).all()


# 256-wide tiles of 256 rows: 9 of them (8 splits fill 74 pairs), 3 x 2 with remainders, one (a single tile of 128 rows), 3 x 199 (more units
# than CTAs with splits), bands of 12 row tiles with a shorter last one
@pytest.mark.parametrize("M,N,Kd", [(768, 768, 4096), (700, 510, 2056), (100, 130, 1000), (6301, 712, 1000), (7000, 8200, 1544)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False)])
def test_splits_and_bands(M, N, Kd, trans_a, trans_b):
    pad = -N % 8
    a = _mk((Kd, M) if trans_a else (M, Kd), 1, (-M % 8) if trans_a else 0)
    b = _mk((N, Kd) if trans_b else (Kd, N), 2, 0 if trans_b else pad, 1 / math.sqrt(Kd))
    ref = (a.t() if trans_a else a).float() @ (b.t() if trans_b else b).float()
    for bn, splits in ((0, 0), (128, 1), (256, 1), (128, 2), (256, 3), (256, 8)):
        out = torch.full((M, N + pad), 7.0, device="cuda", dtype=torch.bfloat16)
        K.gemm(a, b, out[:, :N], trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
        _close(out[:, :N], ref)
        assert (out[:, N:] == 7.0).all()
        again = torch.empty_like(out)
        K.gemm(a, b, again[:, :N], trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
        assert torch.equal(out[:, :N], again[:, :N])


@pytest.mark.parametrize("M,N,Kd", [(512, 256, 2048), (6301, 709, 1000), (300, 131, 72), (130, 64, 4096)])
@pytest.mark.parametrize("what", ["bias", "residual", "accumulate", "gelu with its derivative", "act'"])
def test_epilogue(M, N, Kd, what):
    pad = -N % 8
    a, w = _mk((M, Kd), 3), _mk((N, Kd), 4, 0, 1 / math.sqrt(Kd))
    x = _mk((M, N), 5, pad)
    bias = _mk((1, N + pad), 6).reshape(-1)[:N]
    v = a.float() @ w.float().t()
    out = torch.full((M, N + pad), 7.0, device="cuda", dtype=torch.bfloat16)
    o = out[:, :N]
    if what == "bias":
        K.gemm(a, w, o, trans_b=True, bias=bias)
        ref = v + bias.float()
    elif what == "residual":
        K.gemm(a, w, o, trans_b=True, bias=bias, residual=x)
        ref = v + bias.float() + x.float()
    elif what == "accumulate":
        o.copy_(x)
        K.gemm(a, w, o, trans_b=True, accumulate=True)
        ref = v + x.float()
    elif what == "act'":
        K.gemm(a, w, o, trans_b=True, aux_in=x, act_bwd="mul")
        ref = v * x.float()
    else:
        slope = torch.full_like(out, 7.0)
        K.gemm(a, w, o, trans_b=True, bias=bias, act="gelu_tanh_d", aux_out=slope[:, :N])
        arg = (v + bias.float()).requires_grad_(True)
        y = R.ACTIVATIONS["gelu_tanh"](arg)
        (want,) = torch.autograd.grad(y.sum(), arg)
        assert ((slope[:, :N].float() - want).abs() <= 2.0 ** -6).all() and (slope[:, N:] == 7.0).all()   # slope in bf16, steep by 1.2
        ref = y.detach()
        assert ((o.float() - ref).abs() <= 2.0 ** -7 * ref.abs() + 2.0 ** -7).all()
        return
    _close(o, ref, v, v + bias.float())
    assert (out[:, N:] == 7.0).all()
