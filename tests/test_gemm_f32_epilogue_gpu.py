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
