"""fp32 GEMM kernels against fp64, at tile edges, remainders, every layout, split and epilogue."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200 import ops
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


@pytest.mark.parametrize("M,N,Kd", [(1, 1, 1), (1, 769, 3071), (2, 130, 768), (3, 50, 33), (8, 5000, 260), (9, 65, 17),
                                    (23, 1152, 384), (33, 63, 40), (64, 64, 16), (129, 127, 500), (509, 768, 768),
                                    (1024, 256, 1024)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("pad", [0, 3])
def test_layouts(M, N, Kd, trans_a, trans_b, pad):
    a, b = _mk((Kd, M) if trans_a else (M, Kd), 1, pad), _mk((N, Kd) if trans_b else (Kd, N), 2, pad)
    a2, b2 = (a.t() if trans_a else a), (b.t() if trans_b else b)
    ref, bound = a2.double() @ b2.double(), _bound(a2, b2, Kd)
    for bn in (0, 32, 64, 128):
        for splits in (0, 1, 3):
            out = torch.full((M, N + pad), float("nan"), device="cuda")[:, :N]
            K.gemm(a, b, out, trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
            assert ((out.double() - ref).abs() <= bound).all(), (bn, splits)
            first = out.clone()
            K.gemm(a, b, out, trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
            assert torch.equal(out, first)


@pytest.mark.parametrize("M", [1, 7, 40, 300])
@pytest.mark.parametrize("N", [64, 131])
@pytest.mark.parametrize("act", [None, "relu", "gelu_tanh", "quick_gelu", "silu"])
def test_epilogue(M, N, act):
    a, w, bias = _mk((M, 200), 3), _mk((N, 200), 4) * 0.1, _mk((1, N), 5).reshape(-1)
    res, old = _mk((M, N), 6), _mk((M, N), 7)
    out, pre = old.clone(), torch.empty(M, N, device="cuda")
    K.gemm(a, w, out, trans_b=True, bias=bias, residual=res, aux_out=pre, act=act, accumulate=True, alpha=0.5)
    v = 0.5 * (a.double() @ w.double().t()) + bias.double()
    ref = R.ACTIVATIONS[act](v) + res.double() + old.double()
    assert ((pre.double() - v).abs() <= _bound(a, w.t(), 200) + 4 * EPS * v.abs()).all()
    assert ((out.double() - ref).abs() <= 3 * _bound(a, w.t(), 200) + 16 * EPS * (ref.abs() + res.abs() + old.abs() + 1)).all()
    if act:
        x = _mk((M, N), 8)
        grad = torch.empty(M, N, device="cuda")
        K.gemm(a, w, grad, trans_b=True, aux_in=x, act_bwd=act)
        xd = x.double().requires_grad_(True)
        R.ACTIVATIONS[act](xd).sum().backward()
        ref = (a.double() @ w.double().t()) * xd.grad
        # act' is within 1.2 in size and a few ulp of fp32
        assert ((grad.double() - ref).abs() <= 1.2 * _bound(a, w.t(), 200) + 64 * EPS * (a.double() @ w.double().t()).abs()).all()


def test_infinities_and_nan_stay_in_their_rows():
    a, w = _mk((40, 64), 9), _mk((96, 64), 10)
    a[3, 5], a[7, 0], w[11, 2] = float("inf"), float("nan"), -float("inf")
    for M in (1, 8, 40):
        x = a[32:32 + M] if M < 40 else a
        out, ref = torch.empty(M, 96, device="cuda"), x.double() @ w.double().t()
        K.gemm(x, w, out, trans_b=True)
        assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(torch.isinf(out), torch.isinf(ref))


@pytest.mark.parametrize("act", ["relu", "gelu_tanh", "quick_gelu", "silu"])
def test_mlp_gradients(act):
    M, D, F = 37, 40, 72
    ts = [_mk((M, D), 11), _mk((F, D), 12) * 0.2, _mk((1, F), 13).reshape(-1), _mk((D, F), 14) * 0.2,
          _mk((1, D), 15).reshape(-1), _mk((M, D), 16)]
    x, w1, b1, w2, b2, r = leaves = [t.contiguous().requires_grad_(True) for t in ts]
    y = ops.mlp(x, w1, b1, w2, b2, act, residual=r)
    dy = _mk((M, D), 17)
    y.backward(dy)
    gs = [t.grad.double() for t in leaves]
    exact = [t.detach().double().requires_grad_(True) for t in leaves]
    X, W1, B1, W2, B2, Rr = exact
    Y = R.ACTIVATIONS[act](X @ W1.t() + B1) @ W2.t() + B2 + Rr
    Y.backward(dy.double())
    # chains of two products of up to 72 terms: relative 2-norm errors of about sqrt(72) eps each
    for got, want in zip([y.double()] + gs, [Y] + [t.grad for t in exact]):
        assert float((got - want).norm().detach() / want.norm().detach()) < 8 * math.sqrt(72) * EPS
