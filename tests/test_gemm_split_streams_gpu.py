"""Split products of bf16 on several streams at once: no CTA of one waits for CTAs that the other keeps from an SM, so both give the bits
that they give one after the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200 import _native as N
from dart_pytorch_b200.ops import kernels as K


def _mk(shape, seed):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).bfloat16()


# pairs of CTAs beside pairs, and beside single CTAs (an fp32 output), each with a CTA on nearly every SM
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(768, 768, 8192), (1536, 1280, 2048), (640, 900, 4104)])
def test_two_streams(shape, out_dtype):
    M, N_, Kd = shape
    streams = [torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-1)]
    a, b = [_mk((Kd, M), 2 * i) for i in range(2)], [_mk((Kd, N_ + -N_ % 8), 2 * i + 1)[:, :N_] for i in range(2)]
    dtypes = (torch.bfloat16, out_dtype)

    def product(i, splits):
        out = torch.empty(M, N_, device="cuda", dtype=dtypes[i])
        return K.gemm(a[i], b[i], out, trans_a=True, bn=256 if i == 0 else 128, splits=splits)
    for splits in (4, 8):
        want = [product(i, splits) for i in range(2)]
        ref = [(a[i].double().t() @ b[i].double()) for i in range(2)]
        torch.cuda.synchronize()
        got = [[], []]
        for _ in range(30):
            for i, s in enumerate(streams):
                with torch.cuda.stream(s):
                    got[i].append(product(i, splits))
        torch.cuda.synchronize()
        for i in range(2):
            assert float((want[i].double() - ref[i]).norm() / ref[i].norm()) < 4e-3
            for out in got[i]:
                assert torch.equal(out, want[i]), (i, splits)
    N.raise_on_device_error()
