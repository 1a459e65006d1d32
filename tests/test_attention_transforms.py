"""Attention under forward-mode derivatives and function transforms: refused by the autograd functions, never computed without them."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from dart_pytorch_b200.nn.attention import MultiHeadAttention
from dart_pytorch_b200.ops import flash as A


@pytest.fixture
def no_kernel(monkeypatch):
    monkeypatch.setattr(A, "attn_f32", lambda q, k, v, o, *a, **kw: o.zero_())


@pytest.mark.parametrize("grad_mode", [True, False])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_f32_tangents_are_refused(no_kernel, grad_mode, which):
    ts = [torch.randn(1, 2, 4, 8) for _ in range(3)]
    with torch.set_grad_enabled(grad_mode), fwd.dual_level():
        ts[which] = fwd.make_dual(ts[which], torch.ones(1, 2, 4, 8))
        with pytest.raises(NotImplementedError):
            A.attention_bhsd(*ts, causal=True)
        with pytest.raises(NotImplementedError):
            A.attention_tokens(*(t.reshape(8, 8) for t in ts), 1, 8, 8, 1, 1, 8)


def test_f32_packed_tangents_are_refused(no_kernel):
    with fwd.dual_level(), pytest.raises(NotImplementedError):
        A.attention_packed(fwd.make_dual(torch.randn(4, 48), torch.ones(4, 48)), 1, 4, 2, 2, 8)


def test_f32_transforms_are_refused(no_kernel):
    q = torch.randn(1, 2, 4, 8)

    def attend(x):
        return A.attention_bhsd(x, q, q, causal=True)
    for call in (lambda: torch.func.vmap(attend)(torch.stack([q, q])), lambda: torch.func.jvp(attend, (q,), (q,)),
                 lambda: torch.func.grad(lambda x: attend(x).sum())(q)):
        with pytest.raises(RuntimeError):
            call()


def test_without_transforms_nothing_is_saved(no_kernel, monkeypatch):
    monkeypatch.setattr(A.AttentionF32Fn, "apply", None)
    q = torch.randn(1, 2, 4, 8)
    assert A.attention_bhsd(q, q, q, causal=True).shape == q.shape


@pytest.mark.gpu
@pytest.mark.parametrize("Sq", [1, 2])
def test_cached_bf16_tangents_are_refused(Sq):
    att = MultiHeadAttention(128, 2, device="cuda", dtype=torch.bfloat16)
    q, k = (torch.randn(n, 128, device="cuda", dtype=torch.bfloat16) for n in (2 * Sq, 18))
    k3 = k.view(2, 9, 128)
    with torch.no_grad(), fwd.dual_level(), pytest.raises(NotImplementedError):
        att._attend_tokens(fwd.make_dual(q, torch.ones_like(q)), k3, k3, 2, Sq, 9, Sq > 1, 9 - Sq, None)
