"""Norms over many rows and long cross-entropy rows, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K

BF = torch.bfloat16


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("rows", [4735, 4736, 4737, 9001])
@pytest.mark.parametrize("D", [8, 256, 264, 768, 1000, 1024, 1032, 1536, 1544, 2048, 2056])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("dres", [False, True])
def test_norm(rows, D, rms, dres):
    g = torch.Generator(device="cuda").manual_seed(D)
    x, dy, dr = (torch.randn(rows, D, device="cuda", generator=g).to(BF) for _ in range(3))
    gamma, beta = (torch.randn(D, device="cuda", generator=g).to(BF) for _ in range(2))
    X, G, B = x.double().requires_grad_(True), gamma.double().requires_grad_(True), beta.double().requires_grad_(True)
    if rms:
        y, rstd = K.rmsnorm_fwd(x, gamma, 1e-5)
        dx, dg = K.rmsnorm_bwd(x, dy, gamma, rstd, dres=dr if dres else None)
        Y = X * torch.rsqrt((X * X).mean(-1, keepdim=True) + 1e-5) * G
    else:
        y, mean, rstd = K.layernorm_fwd(x, gamma, beta, 1e-5)
        dx, dg, db = K.layernorm_bwd(x, dy, gamma, mean, rstd, dres=dr if dres else None)
        Y = torch.nn.functional.layer_norm(X, (D,), G, B, 1e-5)
    Y.backward(dy.double())
    # fp32 inside, one rounding to bf16 at the end: no element is off by more than its 2^-8, so the norm is not either
    assert _rel(y, Y.detach()) < 2 ** -8
    assert _rel(dx, X.grad + (dr.double() if dres else 0)) < 2 ** -8
    assert _rel(dg, G.grad) < 2 ** -8
    if not rms:
        assert _rel(db, B.grad) < 2 ** -8


@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("V", [8184, 8192, 8193, 16400, 50257])
def test_cross_entropy_rows(dtype, V):
    rows, pad = 5, (V + 127) // 128 * 128
    buf = (torch.randn(rows, pad, device="cuda") * 4).to(dtype)
    buf[1, :V - 3] = float("-inf")                    # weight at the very end only
    buf[2, 64:8000] = float("-inf")                   # whole stretches without any
    buf[3, 77] = float("nan")
    buf[4, 5] = 300.0
    t = torch.tensor([0, V - 1, 3, 9, 5], device="cuda")
    loss, lse = K.ce_fwd(buf, t, V)
    want = torch.logsumexp(buf[:, :V].double(), -1)
    keep = torch.tensor([0, 1, 2, 4], device="cuda")
    assert torch.isnan(loss[3]) and torch.isnan(lse[3])
    assert torch.allclose(lse[keep].double(), want[keep], rtol=1e-6, atol=1e-5)
    picked = buf[keep].double().gather(1, t[keep, None])[:, 0]
    assert torch.allclose(loss[keep].double(), want[keep] - picked, rtol=1e-5, atol=3e-5)
