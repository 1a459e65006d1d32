"""Infinities and NaN in cached single-token attention: what softmax and the weighted sum make of them, at every key of a chunk."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.nn.attention import MultiHeadAttention

INF, NAN = float("inf"), float("nan")


def _check(H, Hkv, hd, q, k, v):
    B, Sk = k.shape[:2]
    att = MultiHeadAttention(H * hd, H, num_kv_heads=Hkv, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        got = att._attend_tokens(q, k, v, B, 1, Sk, False, Sk - 1, None).double().view(B, H, hd)
    kd, vd = (t.double().view(B, Sk, Hkv, hd).transpose(1, 2).repeat_interleave(H // Hkv, 1) for t in (k, v))
    w = (torch.einsum("bhd,bhjd->bhj", q.double().view(B, H, hd), kd) / math.sqrt(hd)).softmax(-1)
    # a key of weight zero adds nothing but where its value is not finite
    want = torch.where((w == 0)[..., None] & vd.isfinite(), 0.0, w[..., None] * vd).sum(2)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    fin = want.isfinite()
    # (rounded once to bf16, weights by fast exponentials)
    assert (got[fin] - want[fin]).abs().max().item() <= 2.0 ** -7 * max(1.0, want[fin].abs().max().item()) if fin.any() else True


def _inputs(B, H, Hkv, hd, Sk):
    g = torch.Generator(device="cuda").manual_seed(Sk)

    def make(*s):
        return torch.randn(*s, device="cuda", generator=g).bfloat16()
    q = make(B, H * hd)
    q.view(B, H, hd)[..., 3] = 1.0
    return q, make(B, Sk, Hkv * hd), make(B, Sk, Hkv * hd)


SHAPES = [(2, 4, 1, 64), (1, 8, 2, 128), (2, 2, 2, 64), (1, 8, 1, 128)]
LENGTHS = [2, 15, 17, 65, 129, 1000, 5000]


@pytest.mark.parametrize("B,H,Hkv,hd", SHAPES)
@pytest.mark.parametrize("Sk", LENGTHS)
@pytest.mark.parametrize("where", ["first", "last", "middle"])
@pytest.mark.parametrize("x", [INF, -INF, NAN])
def test_values(B, H, Hkv, hd, Sk, where, x):
    q, k, v = _inputs(B, H, Hkv, hd, Sk)
    v[:, {"first": 0, "last": -1, "middle": Sk // 2}[where], 5] = x
    _check(H, Hkv, hd, q, k, v)


@pytest.mark.parametrize("B,H,Hkv,hd", SHAPES)
@pytest.mark.parametrize("Sk", LENGTHS)
@pytest.mark.parametrize("keys", [slice(0, 1), slice(-1, None), slice(0, 64), slice(-200, None), slice(1, None), slice(0, -1)])
def test_scores_of_minus_infinity(B, H, Hkv, hd, Sk, keys):
    q, k, v = _inputs(B, H, Hkv, hd, Sk)
    if len(range(Sk)[keys]) == Sk:
        keys = slice(1, None)
    k.view(B, Sk, Hkv, hd)[:, keys, :, 3] = -INF
    _check(H, Hkv, hd, q, k, v)


@pytest.mark.parametrize("B,H,Hkv,hd", SHAPES)
@pytest.mark.parametrize("Sk", LENGTHS)
@pytest.mark.parametrize("x", [INF, NAN])
def test_keys_and_queries_that_make_nan(B, H, Hkv, hd, Sk, x):
    q, k, v = _inputs(B, H, Hkv, hd, Sk)
    k.view(B, Sk, Hkv, hd)[0, Sk // 2, 0, 3] = x
    _check(H, Hkv, hd, q, k, v)
    q, k, v = _inputs(B, H, Hkv, hd, Sk)
    q[0, 7] = NAN
    _check(H, Hkv, hd, q, k, v)


@pytest.mark.parametrize("Sk", [3, 200, 1000])
def test_no_key_with_a_weight(Sk):
    """Nothing but scores of -inf: zeros, as from the prompt kernel."""
    q, k, v = _inputs(2, 4, 1, 64, Sk)
    k.view(2, Sk, 1, 64)[..., 3] = -INF
    att = MultiHeadAttention(256, 4, num_kv_heads=1, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        assert not att._attend_tokens(q, k, v, 2, 1, Sk, False, Sk - 1, None).any()
