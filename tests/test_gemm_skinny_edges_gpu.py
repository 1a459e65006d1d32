"""Weight-streaming products of few rows where the existing shapes do not reach: the gated form in up to eight parts of K, widths and
strides that leave the 16-byte stores, several waves of tiles."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200 import _native as N
from dart_pytorch_b200.ops import kernels as K


def _mk(shape, seed, pad=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape[0], shape[1] + pad, device="cuda", generator=g) * scale).bfloat16()[:, :shape[1]]


def _swiglu(x, w, out, n, splits=0):
    a = N.GemmArgs()
    a.A, a.B, a.C = x.data_ptr(), w.data_ptr(), out.data_ptr()
    a.lda, a.ldb, a.ldc = x.stride(0), w.stride(0), out.stride(0)
    a.M, a.N, a.K = x.shape[0], n, x.shape[1]
    a.trans_b, a.alpha, a.splits = 1, 1.0, splits
    return N.load().dptb_gemm_skinny_swiglu(ctypes.byref(a), ctypes.c_void_p(N.stream_ptr()))


@pytest.mark.parametrize("M", [1, 32, 33, 64])
@pytest.mark.parametrize("F", [8, 60, 63, 65, 200])
@pytest.mark.parametrize("D", [72, 1000, 4096])
def test_gated_product(M, F, D):
    """Against the product in the same parts, then the gate: the same sums rounded at the same places."""
    pad = 8
    x, w = _mk((M, D), 1, pad), _mk((2 * F, D), 2, pad, D ** -0.5)
    if F == 65:
        x[0, 3], w[1, 2], w[F + 2, 1] = float("inf"), float("nan"), -float("inf")
    for splits in range(1, 9):
        both = torch.empty(M, 2 * F, device="cuda", dtype=torch.bfloat16)
        K.gemm(x, w, both, trans_b=True, splits=splits)
        want = K.swiglu_fwd(both[:, :F].contiguous(), both[:, F:].contiguous())
        out = torch.full((M, F + 5), 7.0, device="cuda", dtype=torch.bfloat16)
        assert _swiglu(x, w, out, F, splits) == 0
        assert torch.equal(out[:, :F].isnan(), want.isnan())
        assert torch.equal(out[:, :F].nan_to_num(3.0), want.nan_to_num(3.0)), splits
        assert (out[:, F:] == 7.0).all()


def test_gated_product_in_waves():
    M, F, D = 17, 64 * 400 + 24, 136                      # 401 tiles, two CTAs an SM
    x, w = _mk((M, D), 3), _mk((2 * F, D), 4, 0, D ** -0.5)
    both = K.gemm(x, w, torch.empty(M, 2 * F, device="cuda", dtype=torch.bfloat16), trans_b=True, splits=1)
    out = torch.empty(M, F, device="cuda", dtype=torch.bfloat16)
    assert _swiglu(x, w, out, F) == 0
    assert torch.equal(out, K.swiglu_fwd(both[:, :F].contiguous(), both[:, F:].contiguous()))


@pytest.mark.parametrize("M", [1, 31, 64])
@pytest.mark.parametrize("width,ld", [(1, 1), (129, 131), (200, 203), (201, 208), (136, 136)])
@pytest.mark.parametrize("splits", [0, 1, 3, 8, 13])
def test_scalar_outputs(M, width, ld, splits):
    """Odd widths, padded rows, and a residual that starts off 16 bytes."""
    D = 1096
    x, w = _mk((M, D), 5), _mk((width, D), 6, 0, D ** -0.5)
    bias = _mk((1, width), 7).reshape(-1)
    res = torch.empty(M * ld + 1, device="cuda", dtype=torch.bfloat16).normal_(generator=torch.Generator(device="cuda").manual_seed(8))
    res = res[1:].view(M, ld)[:, :width]
    out = torch.full((M, ld), 7.0, device="cuda", dtype=torch.bfloat16)
    K.gemm(x, w, out[:, :width], trans_b=True, bias=bias, residual=res, splits=splits)
    ref = x.double() @ w.double().t() + bias.double() + res.double()
    assert ((out[:, :width].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()
    assert (out[:, width:] == 7.0).all()
    whole = K.gemm(x, w, torch.empty(M, width, device="cuda", dtype=torch.bfloat16), trans_b=True, bias=bias,
                   residual=res.contiguous(), splits=splits)
    assert torch.equal(out[:, :width], whole)
