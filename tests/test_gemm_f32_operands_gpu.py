"""fp32 products on tensor cores: operands that are not the sum of three bf16 parts are summed by multiply-adds, their neighbours keep
their bits, and no output is finished twice."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K

EPS = 2.0 ** -24
LAYOUTS = [(False, True), (False, False), (True, False), (True, True)]


def _mk(shape, seed):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def _stored(a, b, trans_a, trans_b):
    """``a [M, K]`` and ``b [K, N]`` as the layout stores them."""
    return (a.t().contiguous() if trans_a else a), (b.t().contiguous() if trans_b else b)


def _gemm(a, b, trans_a, trans_b, **kw):
    sa, sb = _stored(a, b, trans_a, trans_b)
    out = kw.pop("out", None)
    out = torch.empty(a.shape[0], b.shape[1], device="cuda") if out is None else out
    return K.gemm(sa, sb, out, trans_a=trans_a, trans_b=trans_b, **kw)


# from what fills all three parts down to subnormal fp32; the other operand brings the sums back above 2^-100
@pytest.mark.parametrize("small,large", [(1e-29, 1e3), (1e-31, 1e6), (1e-32, 1e6), (1e-33, 1e8), (1e-35, 1e8), (1e-36, 1e12), (1e-37, 1e10),
                                         (1e-38, 1e12), (1e-40, 1e15), (1e-42, 1e30)])
@pytest.mark.parametrize("trans_a,trans_b", LAYOUTS)
@pytest.mark.parametrize("bn,splits", [(1064, 1), (1128, 3), (1064, 8)])
def test_small_against_large(small, large, trans_a, trans_b, bn, splits):
    M, N, Kd = 133, 70, 517
    a, b = (_mk((M, Kd), 1).double() * small).float(), (_mk((Kd, N), 2).double() * large).float()
    for x, y in ((a, b), (b.t().contiguous(), a.t().contiguous())):
        ref = x.double() @ y.double()
        bound = 4.0 * math.sqrt(Kd + 1) * EPS * (x.double().abs() @ y.double().abs()) + 2.0 ** -149 * Kd
        out = _gemm(x, y, trans_a, trans_b, bn=bn, splits=splits)
        assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("trans_a,trans_b", LAYOUTS)
@pytest.mark.parametrize("bn,splits", [(1064, 1), (1128, 2), (1064, 5)])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), 3.4e38, 1e-36, 2.0 ** -149])
def test_neighbours_keep_their_bits(trans_a, trans_b, bn, splits, value):
    M, N, Kd = 150, 140, 400
    a, b = _mk((M, Kd), 3), _mk((Kd, N), 4)
    clean = _gemm(a, b, trans_a, trans_b, bn=bn, splits=splits)
    for rows, cols in (([7], []), ([], [131]), ([0, 149], [66])):
        x, y = a.clone(), b.clone()
        for r in rows:
            x[r, 390] = value
        for c in cols:
            y[3, c] = value
        out, ref = _gemm(x, y, trans_a, trans_b, bn=bn, splits=splits), x.double() @ y.double()
        keep = torch.ones(M, N, dtype=torch.bool, device="cuda")
        keep[rows], keep[:, cols] = False, False
        assert torch.equal(out[keep], clean[keep])
        size = x.double().abs() @ y.double().abs()
        fin = size < 3e38                                   # (between that and infinity a sum may overflow on its way)
        bad = ~size.isfinite()
        assert torch.equal(out.isnan()[bad], ref.isnan()[bad]) and torch.equal(out.isinf()[bad], ref.isinf()[bad])
        bound = 4.0 * math.sqrt(Kd + 1) * EPS * size
        assert ((out.double() - ref).abs()[fin] <= bound[fin]).all()


@pytest.mark.parametrize("bn,splits", [(1064, 1), (1128, 4)])
@pytest.mark.parametrize("N", [140, 141])
def test_every_output_is_finished_once(bn, splits, N):
    """Sums that are added to what is there, with an activation and a saved argument, where every other row is computed again."""
    M, Kd = 130, 300
    a, b, old, bias = _mk((M, Kd), 5), _mk((Kd, N), 6), _mk((M, N), 7), _mk((N,), 8)
    a[::2, 5] = 1e-37
    out, pre = old.clone(), torch.full((M, N), 7.0, device="cuda")
    _gemm(a, b, False, True, out=out, bias=bias, act="relu", aux_out=pre, accumulate=True, bn=bn, splits=splits)
    v = a.double() @ b.double() + bias.double()
    bound = 4.0 * math.sqrt(Kd + 1) * EPS * (a.double().abs() @ b.double().abs()) + 4 * EPS * (v.abs() + old.double().abs() + 1)
    assert ((pre.double() - v).abs() <= bound).all()
    assert ((out.double() - (v.relu() + old.double())).abs() <= 2 * bound).all()


@pytest.mark.parametrize("Kd", [256, 768, 3072])
@pytest.mark.parametrize("kind", ["normal", "one sign", "exponential"])
def test_no_further_from_fp64(Kd, kind):
    """Also where all products have one sign, so that truncations in the accumulator would add up."""
    M, N = 256, 256
    a, w = _mk((M, Kd), 11), _mk((N, Kd), 12)
    if kind == "one sign":
        a, w = a.abs(), w.abs()
    elif kind == "exponential":
        a, w = a.exp(), w.exp()
    ref = a.double() @ w.double().t()

    def error(bn, splits):
        out = torch.empty(M, N, device="cuda")
        K.gemm(a, w, out, trans_b=True, bn=bn, splits=splits)
        return float((out.double() - ref).norm() / ref.norm())
    got = {(bn, s): error(bn, s) for bn in (1064, 1128) for s in (1, 2, 4)}
    plain = error(64, 1)
    print(kind, Kd, {k: f"{v:.2e}" for k, v in got.items()}, f"{plain:.2e}")
    assert max(got.values()) <= plain


# the tile and the parts of K that multiply-adds would take
@pytest.mark.parametrize("M,N,Kd,bn,splits", [(509, 768, 768, 64, 6), (256, 256, 1024, 32, 16), (23, 384, 384, 32, 6),
                                               (1024, 256, 1024, 64, 8), (200, 512, 640, 32, 10)])
def test_one_sign_against_multiply_adds_in_parts(M, N, Kd, bn, splits):
    def error(**kw):
        total = 0.0
        for seed in range(4):
            a, w = _mk((M, Kd), 20 + seed).abs(), _mk((N, Kd), 30 + seed).abs()
            out, ref = torch.empty(M, N, device="cuda"), a.double() @ w.double().t()
            K.gemm(a, w, out, trans_b=True, **kw)
            total += float((out.double() - ref).norm() / ref.norm())
        return total
    assert error() <= error(bn=bn, splits=splits)
