"""Weight-streaming products of few rows: where K is cut is part of the result, so the rule is pinned, and every number of parts that a
cluster can hold gives the sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K


def _mk(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, device="cuda", generator=g) * scale).bfloat16()


# (148 SMs: one part while the tiles fill them, parts of at least 8 k-blocks, 16 at most)
@pytest.mark.parametrize("N,Kd,parts", [(11008, 2048, 1), (2048, 5504, 9), (3072, 2048, 4), (2048, 2048, 4), (768, 768, 1),
                                        (1000, 1100, 2), (512, 8448, 16), (128, 500, 1)])
@pytest.mark.parametrize("M", [1, 32, 33])
def test_where_k_is_cut(M, N, Kd, parts):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the rule fills the SMs")
    x, w = _mk((M, Kd), 1), _mk((N, Kd), 2, Kd ** -0.5)
    out = K.gemm(x, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), trans_b=True)
    # each part is one accumulator in fp32, its products in order; the parts are added in order and rounded once
    want = K.gemm(x, w, torch.empty_like(out), trans_b=True, splits=parts)
    assert torch.equal(out, want)


@pytest.mark.parametrize("parts", [1, 2, 3, 7, 8, 9, 11, 16])
@pytest.mark.parametrize("M,N,Kd", [(1, 130, 1400), (40, 1000, 2048)])
def test_parts(M, N, Kd, parts):
    x, w, res = _mk((M, Kd), 3), _mk((N, Kd), 4, Kd ** -0.5), _mk((M, N), 5)
    out = K.gemm(x, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), trans_b=True, residual=res, splits=parts)
    ref = x.double() @ w.double().t() + res.double()
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()
    kb = -(-Kd // 64)                                       # the same as fp32 sums of each part's exact products, to their rounding
    per = -(-kb // parts) * 64
    total = torch.zeros(M, N, device="cuda")
    for k in range(0, Kd, per):
        total += (x[:, k:k + per].double() @ w[:, k:k + per].double().t()).float()
    assert ((out.float() - (total + res.float())).abs() <= 2.0 ** -8 * ref.abs().float() + 1e-4).all()
