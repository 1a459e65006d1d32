"""Heads of other sizes than 64 and 128, read as they are by the forward kernel, against fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import flash


def _want(q, k, v, causal, q_offset):
    """``[B, S, heads, hd]`` operands in fp64."""
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    k, v = (t.repeat_interleave(q.shape[1] // t.shape[1], 1) for t in (k, v))
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        i, j = torch.arange(s.shape[-2], device="cuda")[:, None] + q_offset, torch.arange(s.shape[-1], device="cuda")
        s = s.masked_fill(j > i, float("-inf"))
    return (s.softmax(-1) @ v).transpose(1, 2)


@pytest.mark.parametrize("hd", [8, 24, 32, 56, 72, 120])
@pytest.mark.parametrize("B,Sq,Sk,H,Hkv,causal", [(1, 1, 1, 1, 1, False), (2, 127, 127, 3, 3, True), (3, 129, 129, 4, 2, False),
                                                  (2, 300, 300, 2, 1, True), (2, 5, 260, 4, 4, True)])
@pytest.mark.parametrize("nan_head", [False, True])
def test_forward(hd, B, Sq, Sk, H, Hkv, causal, nan_head):
    g = torch.Generator(device="cuda").manual_seed(hd)
    q, k, v = (torch.randn(B, S, n, hd, device="cuda", generator=g).bfloat16() for S, n in ((Sq, H), (Sk, Hkv), (Sk, Hkv)))
    if nan_head:                 # a head's neighbours in memory are none of its business
        k[:, :, -1], v[:, :, -1] = float("nan"), float("inf")
    keep = H // Hkv * (Hkv - 1) if nan_head else H
    with torch.no_grad():
        o = flash.attention_tokens(q.view(B * Sq, -1), k.view(B * Sk, -1), v.view(B * Sk, -1), B, Sq, Sk, H, Hkv, hd, causal,
                                   Sk - Sq).view(B, Sq, H, hd)[:, :, :keep]
    want = _want(q, k, v, causal, Sk - Sq)[:, :, :keep]
    # probabilities and the result rounded to bf16: up to 2^-8 each, about half of it in root mean square
    assert o.numel() == 0 or float((o.double() - want).norm() / want.norm()) < 2 ** -8 * 1.5


def test_unaligned_rows_take_the_padding_path():
    B, S, H, hd = 2, 70, 2, 32
    x = torch.randn(B * S, 3 * H * hd + 1, device="cuda").bfloat16()[:, 1:]
    q, k, v = x[:, :64], x[:, 64:128], x[:, 128:]
    with torch.no_grad():
        a = flash.attention_tokens(q, k, v, B, S, S, H, H, hd)
        b = flash.attention_tokens(q.contiguous(), k.contiguous(), v.contiguous(), B, S, S, H, H, hd)
    assert float((a.float() - b.float()).norm() / b.float().norm()) < 1e-2
