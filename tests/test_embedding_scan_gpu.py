"""The scanned embedding gradient: the same additions in the same order as the sorted one, so the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,V,D", [(1, 1, 1), (31, 3, 8), (33, 65, 100), (257, 5, 264), (1024, 65, 256), (603, 320, 128),
                                   (2048, 50257, 770), (2048, 1, 64)])
def test_scan_equals_sorted(monkeypatch, dtype, n, V, D):
    g = torch.Generator(device="cuda").manual_seed(n)
    idx = torch.randint(0, V, (n,), device="cuda", generator=g)
    idx[torch.rand(n, device="cuda", generator=g) < 0.05] = V       # out of range: skipped
    idx[n // 2] = -1
    dout = torch.randn(n, D, device="cuda", generator=g).to(dtype)
    start = torch.randn(V, D, device="cuda", generator=g).to(dtype)
    got, want = start.clone(), start.clone()
    assert n <= K.EMBED_SCAN_TOKENS
    K.embedding_bwd(got, idx, dout)
    monkeypatch.setattr(K, "EMBED_SCAN_TOKENS", 0)
    K.embedding_bwd(want, idx, dout)
    assert torch.equal(got, want)
    exact = start.double().index_add(0, idx.clamp(0, V - 1), dout.double() * ((idx >= 0) & (idx < V))[:, None])
    # a sum of up to 2048 fp32 terms of about 1, rounded once to the dtype
    assert torch.allclose(got.double(), exact, rtol=2 ** -8 if dtype == torch.bfloat16 else 1e-5, atol=1e-3)
