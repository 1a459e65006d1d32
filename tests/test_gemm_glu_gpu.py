"""The gated product against the product, then the gate: the same sums, rounded at the same places, so the same bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200 import _native as N
from dart_pytorch_b200.ops import kernels as K


def _call(x, w, out, n):
    a = N.GemmArgs()
    a.A, a.B, a.C = x.data_ptr(), w.data_ptr(), out.data_ptr()
    a.lda, a.ldb, a.ldc = x.stride(0), w.stride(0), out.stride(0)
    a.M, a.N, a.K = x.shape[0], n, x.shape[1]
    a.trans_b, a.alpha = 1, 1.0
    return N.load().dptb_gemm_swiglu(ctypes.byref(a), ctypes.c_void_p(N.stream_ptr()))


# tiles are 256 rows x 128 columns: one row more than a row tile, the edges of pairs of them, odd pairs; widths around 64 and 128
@pytest.mark.parametrize("M", [129, 256, 257, 700])
@pytest.mark.parametrize("F,D", [(8, 64), (56, 72), (128, 64), (136, 200), (328, 128), (1000, 256)])
@pytest.mark.parametrize("pad", [0, 8])
def test_same_bits(M, F, D, pad):
    g = torch.Generator(device="cuda").manual_seed(M + F)
    x = torch.randn(M, D + pad, device="cuda", generator=g).bfloat16()[:, :D]
    w = torch.randn(2 * F, D + pad, device="cuda", generator=g).bfloat16()[:, :D]
    if pad:
        x[5, 3], w[1, 2], w[F + 2, 1] = float("inf"), float("nan"), -float("inf")
    both = torch.empty(M, 2 * F, device="cuda", dtype=torch.bfloat16)
    K.gemm(x, w, both, trans_b=True, splits=1)
    want = K.swiglu_fwd(both[:, :F], both[:, F:])
    out = torch.full((M, F + pad), 7.0, device="cuda", dtype=torch.bfloat16)
    assert _call(x, w, out, F) == 0
    assert torch.equal(out[:, :F].nan_to_num(3.0), want.nan_to_num(3.0)) and torch.equal(out[:, :F].isnan(), want.isnan())
    assert (out[:, F:] == 7.0).all()


def test_declines():
    x, w = torch.zeros(200, 64, device="cuda").bfloat16(), torch.zeros(40, 64, device="cuda").bfloat16()
    out = torch.full((200, 20), 7.0, device="cuda", dtype=torch.bfloat16)
    assert _call(x, w, out, 20) == K.ERR_UNSUPPORTED          # a width that is no multiple of 8
    assert _call(x[:128], w, out[:128], 16) == K.ERR_UNSUPPORTED   # one row tile
    assert (out == 7.0).all()
