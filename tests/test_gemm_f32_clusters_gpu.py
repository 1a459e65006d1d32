"""fp32 products whose parts of K meet in a cluster, launched one behind the other without a wait: tiles whose lanes finish apart (odd
rows, ragged columns, outputs that are computed again) give the bits of a launch by itself, every time."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200 import _native as N
from dart_pytorch_b200.ops import kernels as K


def _mk(shape, seed):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


@pytest.mark.parametrize("M,N_,Kd", [(23, 384, 512), (125, 67, 513), (129, 130, 1030), (509, 770, 768), (1, 1, 640)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False)])
@pytest.mark.parametrize("nonfinite", [False, True])
def test_back_to_back(M, N_, Kd, trans_a, trans_b, nonfinite):
    a, b = _mk((Kd, M) if trans_a else (M, Kd), 1), _mk((N_, Kd) if trans_b else (Kd, N_), 2)
    if nonfinite:
        a[a.shape[0] // 2, a.shape[1] // 3] = float("inf")
        b[0, b.shape[1] - 1] = float("nan")
    for bn in (1064, 1128):
        for splits in (2, 3, 5, 8):
            first = K.gemm(a, b, torch.empty(M, N_, device="cuda"), trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
            torch.cuda.synchronize()
            outs = [torch.full_like(first, 7.0) for _ in range(20)]
            for out in outs:
                K.gemm(a, b, out, trans_a=trans_a, trans_b=trans_b, bn=bn, splits=splits)
            for out in outs:
                assert torch.equal(out.view(torch.int32), first.view(torch.int32)), (bn, splits)
    N.raise_on_device_error()
