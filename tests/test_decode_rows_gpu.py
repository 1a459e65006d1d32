"""Split-key decode attention against fp64 at the edges of its rounds, splits and head groups."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import decode as D


def _want(q, k, v, H, Hkv, hd):
    B, Sk = k.shape[:2]
    k, v = (t.double().reshape(B, Sk, Hkv, hd).transpose(1, 2).repeat_interleave(H // Hkv, 1) for t in (k, v))
    s = q.double().reshape(B, H, 1, hd) @ k.transpose(-1, -2) / math.sqrt(hd)
    return (s.softmax(-1) @ v).reshape(B, H * hd)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("H,Hkv", [(1, 1), (2, 1), (6, 2), (4, 1), (7, 1), (16, 2)])
@pytest.mark.parametrize("Sk,splits", [(1, 0), (15, 1), (16, 2), (17, 1), (63, 0), (65, 3), (257, 5), (1000, 0)])
def test_against_fp64(hd, H, Hkv, Sk, splits):
    g = torch.Generator(device="cuda").manual_seed(Sk)
    B = 3
    q = torch.randn(B, H * hd, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(B, Sk + 2, Hkv * hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    k[:, Sk:], v[:, Sk:] = float("nan"), float("nan")               # rows nobody may read
    o = D.attn_decode(q, k, v, B, 1, Sk, H, Hkv, hd, Sk - 1, splits=splits)
    want = _want(q, k[:, :Sk], v[:, :Sk], H, Hkv, hd)
    # weights and sums carry 24 bits: the result's own rounding is what shows, at most 2^-8 of each element
    assert float((o.double() - want).norm() / want.norm()) < 2.0 ** -8


def test_large_scores_and_infinite_values():
    B, H, hd, Sk = 2, 4, 64, 100
    q = torch.randn(B, H * hd, device="cuda").bfloat16() * 50
    k, v = (torch.randn(B, Sk, hd, device="cuda").bfloat16() for _ in range(2))
    o = D.attn_decode(q, k, v, B, 1, Sk, H, 1, hd, Sk - 1)
    want = _want(q, k, v, H, 1, hd)
    assert torch.isfinite(o).all() and float((o.double() - want).norm() / want.norm()) < 2.0 ** -8
    v[0, 3, 5] = float("inf")
    q = torch.zeros_like(q)                                          # equal weights: every head sees it
    o = D.attn_decode(q, k, v, B, 1, Sk, H, 1, hd, Sk - 1).view(B, H, hd)
    assert (o[0, :, 5] == float("inf")).all() and torch.isfinite(o[0, :, 6:]).all() and torch.isfinite(o[1]).all()
