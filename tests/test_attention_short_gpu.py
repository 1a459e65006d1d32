"""bf16 attention over sequences of one query tile, where a CTA takes two heads at a time once there are more heads than SMs: the same
bits as of the same sequences one at a time (a head has a CTA to itself then), and the formula in fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200 import ops


def _exact(q, k, v, causal):
    g = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(g, 1), v.repeat_interleave(g, 1)
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        i = torch.arange(q.shape[2], device=q.device)[:, None] + k.shape[2] - q.shape[2]
        s = s.masked_fill(torch.arange(k.shape[2], device=q.device)[None] > i, float("-inf"))
    return s.softmax(-1) @ v


# An odd number of heads in all (the last CTA has one), one round and several, grouped queries, both ends of the tile, keys of more than
# one tile.  Bound: the output is rounded to 8 bits, and each weight of the sum is, independently.
@pytest.mark.parametrize("B,H,Hkv,S,causal", [(51, 3, 3, 128, True), (64, 12, 12, 119, False), (200, 1, 1, 1, True), (90, 8, 2, 37, True),
                                              (149, 1, 1, 127, False), (300, 5, 1, 128, False)])
def test_packed(B, H, Hkv, S, causal):
    for hd in (64, 32, 40):
        g = torch.Generator(device="cuda").manual_seed(S + hd)
        x = torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda", generator=g).bfloat16()
        with torch.no_grad():
            o = ops.attention_packed(x, B, S, H, Hkv, hd, causal)
            for b in (0, B // 2, B - 1):
                rows = slice(b * S, (b + 1) * S)
                assert torch.equal(o[rows], ops.attention_packed(x[rows], 1, S, H, Hkv, hd, causal))
        q, k, v = x.double().split([H * hd, Hkv * hd, Hkv * hd], 1)
        ref = _exact(*(t.reshape(B, S, -1, hd).transpose(1, 2) for t in (q, k, v)), causal).transpose(1, 2).reshape(B * S, -1)
        assert float((o.double() - ref).norm() / ref.norm()) < 2 ** -8


@pytest.mark.parametrize("B,H,Hkv,S,Sk,causal", [(40, 4, 2, 70, 300, True), (77, 2, 2, 128, 257, False), (151, 1, 1, 5, 129, True)])
def test_more_keys_than_queries(B, H, Hkv, S, Sk, causal):
    g = torch.Generator(device="cuda").manual_seed(Sk)
    q, k, v = (torch.randn(B, h, s, 64, device="cuda", generator=g).bfloat16() for h, s in ((H, S), (Hkv, Sk), (Hkv, Sk)))
    with torch.no_grad():
        o = ops.attention(q, k, v, causal=causal, q_offset=Sk - S)
        assert torch.equal(o[:1], ops.attention(q[:1], k[:1], v[:1], causal=causal, q_offset=Sk - S))
        assert torch.equal(o[-1:], ops.attention(q[-1:], k[-1:], v[-1:], causal=causal, q_offset=Sk - S))
    ref = _exact(q.double(), k.double(), v.double(), causal)
    assert float((o.double() - ref).norm() / ref.norm()) < 2 ** -8


def test_gradients():
    """The backward pass reads the log-sum-exp that the forward left."""
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k, v = (torch.randn(52, 3, 101, 64, device="cuda", generator=g).bfloat16().requires_grad_(True) for _ in range(3))
    do = torch.randn(52, 3, 101, 64, device="cuda", generator=g).bfloat16()
    got = torch.autograd.grad(ops.attention(q, k, v, causal=True), (q, k, v), do)
    d = [t.detach().double().requires_grad_(True) for t in (q, k, v)]
    for a, b in zip(got, torch.autograd.grad(_exact(*d, True), d, do.double())):
        assert float((a.double() - b).norm() / b.norm()) < 2 ** -7
