"""What the fp32 GEMM does after the product, against fp64, in each of its kernels: rows that stream the weight (up to 8 rows,
256 terms and more), tiles, and the fold of a split K."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K
from dart_pytorch_b200.ops import reference as R

EPS = 2.0 ** -24


def _mk(shape, seed, pad=0):
    """A matrix whose rows are ``pad`` elements apart from one another beyond their length."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape[0], shape[1] + pad, device="cuda", generator=g)[:, :shape[1]]


def _bound(a, b, K_):
    """Largest error of a sum of K products, each rounded once: ``K eps sum |a||b|`` bounds it; 4 sqrt(K) is far out in
    the tail of independent roundings."""
    return 4.0 * math.sqrt(K_ + 1) * EPS * (a.double().abs() @ b.double().abs()) + 1e-30


@pytest.mark.parametrize("M,splits", [(1, 0), (3, 0), (8, 0), (40, 1), (40, 3)])
@pytest.mark.parametrize("Kd", [64, 771])
@pytest.mark.parametrize("pad", [0, 3])
def test_gelu_with_its_derivative(M, splits, Kd, pad):
    """``gelu_tanh_d`` without an ``aux_out`` is GELU; with one the derivative goes there, and ``mul`` takes it back."""
    N = 66
    a, w, bias = _mk((M, Kd), 1, pad), _mk((N, Kd), 2, pad) * (2.0 / math.sqrt(Kd)), _mk((1, N), 3).reshape(-1)
    v = (a.double() @ w.double().t() + bias.double()).requires_grad_(True)
    gelu = R.ACTIVATIONS["gelu_tanh"](v)
    (slope,) = torch.autograd.grad(gelu.sum(), v)
    # both are within 1.2 of the value's error, and a few roundings of terms of their size
    tol = 1.2 * _bound(a, w.t(), Kd) + 32 * EPS * (1 + v.detach().abs())
    out, out2, d = (torch.full((M, N + pad), float("nan"), device="cuda")[:, :N] for _ in range(3))
    K.gemm(a, w, out, trans_b=True, bias=bias, act="gelu_tanh_d", splits=splits)
    K.gemm(a, w, out2, trans_b=True, bias=bias, act="gelu_tanh_d", aux_out=d, splits=splits)
    assert ((out.double() - gelu.detach()).abs() <= tol).all() and torch.equal(out, out2)
    assert ((d.double() - slope).abs() <= tol).all()
    back = torch.empty(M, N, device="cuda")
    K.gemm(a, w, back, trans_b=True, aux_in=d, act_bwd="mul", splits=splits)
    want = (a.double() @ w.double().t()) * slope
    assert ((back.double() - want).abs() <= 1.2 * _bound(a, w.t(), Kd) + tol * want.abs() + 4 * EPS * want.abs()).all()


@pytest.mark.parametrize("M,splits", [(1, 0), (2, 0), (3, 0), (5, 0), (8, 0), (9, 0), (9, 3), (70, 3)])
@pytest.mark.parametrize("Kd", [200, 260, 771, 3072])
@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("act", [None, "relu", "gelu_tanh", "quick_gelu", "silu"])
def test_everything_after_the_product(M, splits, Kd, pad, act):
    N = 67
    a, w = _mk((M, Kd), 3, pad), _mk((N, Kd), 4, pad) * (2.0 / math.sqrt(Kd))
    bias = _mk((1, N), 5).reshape(-1)
    if M % 2:
        bias = bias.bfloat16()
    res, old, x = _mk((M, N), 6, pad), _mk((M, N), 7, pad), _mk((M, N), 8, pad)
    behind = torch.full((M, N + pad), 5.0, device="cuda")
    out, pre = behind.clone()[:, :N], behind.clone()[:, :N]
    out.copy_(old)
    K.gemm(a, w, out, trans_b=True, bias=bias, residual=res, aux_out=pre, act=act, accumulate=True, alpha=0.5, splits=splits)
    product = a.double() @ w.double().t()
    v, bound = 0.5 * product + bias.double(), _bound(a, w.t(), Kd)
    ref = R.ACTIVATIONS[act](v) + res.double() + old.double()
    assert ((pre.double() - v).abs() <= bound + 4 * EPS * (v.abs() + bias.abs())).all()
    assert ((out.double() - ref).abs() <= 1.2 * bound + 16 * EPS * (ref.abs() + v.abs() + res.abs() + old.abs() + 1)).all()
    for t in (out, pre):
        assert (t.as_strided((M, N + pad), (N + pad, 1))[:, N:] == 5.0).all()
    if act:
        grad = torch.empty(M, N + pad, device="cuda")[:, :N]
        K.gemm(a, w, grad, trans_b=True, aux_in=x, act_bwd=act, splits=splits)
        xd = x.double().requires_grad_(True)
        R.ACTIVATIONS[act](xd).sum().backward()
        # act' is within 1.2 in size and a few ulp of fp32
        assert ((grad.double() - product * xd.grad).abs() <= 1.2 * bound + 64 * EPS * product.abs()).all()


@pytest.mark.parametrize("M,splits", [(1, 0), (3, 0), (8, 0), (9, 1), (40, 3)])
@pytest.mark.parametrize("Kd", [260, 771])
def test_infinities_and_nan_stay_in_their_rows(M, splits, Kd):
    a, w = _mk((M, Kd), 9), _mk((96, Kd), 10)
    w[11, 2], w[95, Kd - 1] = -float("inf"), float("nan")
    if M > 1:
        a[M - 1, 5], a[1, Kd - 1] = float("inf"), float("nan")
    out, ref = torch.empty(M, 96, device="cuda"), a.double() @ w.double().t()
    K.gemm(a, w, out, trans_b=True, splits=splits)
    assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(torch.isinf(out), torch.isinf(ref))
