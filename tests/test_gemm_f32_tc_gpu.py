"""fp32 GEMM on the tensor cores (operands in three bf16 parts) against fp64: edges of its tiles, k-blocks and parts of K, every
layout, its epilogue, and values that have no three parts."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K
from dart_pytorch_b200.ops import reference as R

EPS = 2.0 ** -24
WIDE, NARROW = 1128, 1064      # tiles of 128 and of 64 columns


def _mk(shape, seed, pad=0):
    """A matrix whose rows are ``pad`` elements apart from one another beyond their length."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape[0], shape[1] + pad, device="cuda", generator=g)[:, :shape[1]]


def _bound(a, b, K_):
    """A k-block's sum meets up to four truncations (2^-23 each) and the blocks one rounding each: within what K roundings of
    2^-24 leave, ``4 sqrt(K)`` far out in their tail."""
    return 4.0 * math.sqrt(K_ + 1) * EPS * (a.double().abs() @ b.double().abs()) + 1e-30


@pytest.mark.parametrize("M,N,Kd", [(1, 1, 1), (9, 1, 63), (127, 63, 64), (128, 64, 65), (129, 65, 129), (23, 127, 400),
                                    (130, 128, 512), (257, 129, 1030)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("pad", [0, 3, 4])
def test_layouts(M, N, Kd, trans_a, trans_b, pad):
    a, b = _mk((Kd, M) if trans_a else (M, Kd), 1, pad), _mk((N, Kd) if trans_b else (Kd, N), 2, pad)
    a2, b2 = (a.t() if trans_a else a), (b.t() if trans_b else b)
    ref, bound = a2.double() @ b2.double(), _bound(a2, b2, Kd)
    for bn in (NARROW, WIDE):
        for splits in (1, 2, 5, 8):
            out = torch.full((M, N + pad), 7.0, device="cuda")
            K.gemm(a, b, out[:, :N], trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
            assert ((out[:, :N].double() - ref).abs() <= bound).all(), (bn, splits)
            assert (out[:, N:] == 7.0).all()
            again = torch.empty_like(out)
            K.gemm(a, b, again[:, :N], trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
            assert torch.equal(out[:, :N], again[:, :N])


@pytest.mark.parametrize("M,N", [(40, 64), (130, 131)])
@pytest.mark.parametrize("act", [None, "relu", "gelu_tanh", "silu"])
def test_epilogue(M, N, act):
    a, w, bias = _mk((M, 320), 3), _mk((N, 320), 4) * 0.1, _mk((1, N), 5).reshape(-1)
    res, old = _mk((M, N), 6), _mk((M, N), 7)
    for bn, splits in ((NARROW, 1), (WIDE, 3)):
        out, pre = old.clone(), torch.empty(M, N, device="cuda")
        K.gemm(a, w, out, trans_b=True, bias=bias, residual=res, aux_out=pre, act=act, accumulate=True, alpha=0.5, bn=bn, splits=splits)
        v = 0.5 * (a.double() @ w.double().t()) + bias.double()
        ref = R.ACTIVATIONS[act](v) + res.double() + old.double()
        assert ((pre.double() - v).abs() <= _bound(a, w.t(), 320) + 4 * EPS * v.abs()).all()
        assert ((out.double() - ref).abs() <= 3 * _bound(a, w.t(), 320) + 16 * EPS * (ref.abs() + res.abs() + old.abs() + 1)).all()


@pytest.mark.parametrize("M,N,Kd", [(300, 256, 256), (256, 300, 1024), (200, 128, 3072)])
@pytest.mark.parametrize("gelu", [False, True])
def test_no_further_from_fp64_than_multiply_adds(M, N, Kd, gelu):
    a, w = _mk((M, Kd), 11), _mk((N, Kd), 12)
    if gelu:
        a = torch.nn.functional.gelu(a)
    ref = a.double() @ w.double().t()

    def error(bn, splits):
        out = torch.empty(M, N, device="cuda")
        K.gemm(a, w, out, trans_b=True, bn=bn, splits=splits)
        return float((out.double() - ref).norm())
    assert max(error(WIDE, 1), error(NARROW, 4)) <= error(64, 1)


@pytest.mark.parametrize("bn,splits", [(NARROW, 1), (WIDE, 3)])
def test_values_without_three_parts(bn, splits):
    M, N, Kd = 40, 96, 330
    a, w = _mk((M, Kd), 9), _mk((N, Kd), 10)
    a[3, 5], a[7, 0], w[11, 2], w[95, Kd - 1] = float("inf"), float("nan"), -float("inf"), float("nan")
    a[20], w[30] = 0.0, 0.0
    a[20, 4], w[30, 4] = 3.402e38, 0.5                       # rounds to infinity in bf16
    out, ref = torch.empty(M, N, device="cuda"), a.double() @ w.double().t()
    ref = ref.float().double()
    K.gemm(a, w, out, trans_b=True, bn=bn, splits=splits)
    assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(torch.isinf(out), torch.isinf(ref))
    assert float(out[20, 30]) == 3.402e38 * 0.5 or abs(float(out[20, 30]) / (3.402e38 * 0.5) - 1) < 2 * EPS
    # magnitudes whose low parts have no bf16: the run of fma
    tiny, x = _mk((M, Kd), 13) * 1e-36, _mk((N, Kd), 14)
    K.gemm(tiny, x, out, trans_b=True, bn=bn, splits=splits)
    bound = 4.0 * math.sqrt(Kd + 1) * EPS * (tiny.double().abs() @ x.double().abs().t())
    assert ((out.double() - tiny.double() @ x.double().t()).abs() <= bound).all()
    K.gemm(torch.zeros_like(a), x, out, trans_b=True, bn=bn, splits=splits)
    assert (out == 0).all()
