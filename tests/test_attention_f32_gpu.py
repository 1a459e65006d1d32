"""fp32 attention kernels against the same formula in fp64: output and gradients, over the edges of their tiles (32 query rows,
64 keys, 8 rows of a kv head for the split form), grouped queries, offsets, odd head sizes and strides."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import flash as A


def _exact(q, k, v, causal, off):
    g = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(g, 1), v.repeat_interleave(g, 1)
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        i = torch.arange(q.shape[2], device=q.device)[:, None] + off
        s = s.masked_fill(torch.arange(k.shape[2], device=q.device)[None] > i, float("-inf"))
    return s.softmax(-1) @ v


# B, H, Hkv, Sq, Sk, hd, causal, offset.  Bound: a product of hd terms and a softmax-weighted sum, each within a few units of
# 2^-24 times the root of its length (1.5e-6 at 64 x 1000); gradients pass two of them.
CASES = [(1, 1, 1, 1, 1, 64, True, 0), (2, 3, 3, 33, 33, 64, True, 0), (1, 2, 2, 32, 64, 32, False, 0), (2, 4, 2, 65, 129, 16, False, 0),
         (1, 12, 12, 1, 510, 64, True, 509), (2, 8, 1, 1, 1000, 128, True, 999), (1, 4, 2, 4, 65, 64, True, 61),
         (1, 4, 2, 5, 70, 64, True, 65), (1, 2, 1, 100, 300, 128, True, 200), (2, 2, 2, 40, 40, 10, True, 0), (1, 2, 2, 31, 63, 7, False, 0),
         (1, 1, 1, 127, 127, 100, True, 0)]


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,hd,causal,off", CASES)
@pytest.mark.parametrize("layout", ["bhsd", "token", "odd"])
def test_attention_f32(B, H, Hkv, Sq, Sk, hd, causal, off, layout):
    g = torch.Generator(device="cuda").manual_seed(Sq * 7 + hd)

    def make(h, s):
        t = torch.randn(B, s, h, hd, device="cuda", generator=g)
        if layout == "bhsd":
            return t.transpose(1, 2).contiguous()
        if layout == "odd":       # rows start at addresses that are no multiple of 16 bytes
            wide = torch.zeros(B, s, h, hd + 3, device="cuda")
            wide[..., 1:hd + 1] = t
            return wide[..., 1:hd + 1].transpose(1, 2)
        return t.transpose(1, 2)
    q, k, v = (make(H, Sq).requires_grad_(True), make(Hkv, Sk).requires_grad_(True), make(Hkv, Sk).requires_grad_(True))
    o = A.attention_bhsd(q, k, v, causal, None, off)
    do = torch.randn(o.shape, device="cuda", generator=g)
    got = torch.autograd.grad(o, (q, k, v), do)
    with torch.no_grad():
        assert torch.equal(A.attention_bhsd(q, k, v, causal, None, off), o)
    d = [t.detach().double().requires_grad_(True) for t in (q, k, v)]
    ref = _exact(*d, causal, off)
    want = torch.autograd.grad(ref, d, do.double())
    for a, b in zip((o.detach(), *got), (ref.detach(), *want)):
        if float(b.norm()) < 1e-6:      # one key: its weight is 1 whatever the score, and the exact dQ and dK are zero
            assert float(a.abs().max()) < 1e-6
        else:
            assert float((a.double() - b).norm() / b.norm()) < 3e-6


@pytest.mark.parametrize("B,S,H,Hkv,hd", [(2, 96, 4, 2, 32), (1, 33, 3, 3, 20)])
def test_packed_f32_is_one_launch_and_matches_separate_operands(B, S, H, Hkv, hd):
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda", generator=g).requires_grad_(True)
    do = torch.randn(B * S, H * hd, device="cuda", generator=g)
    o = A.attention_packed(x, B, S, H, Hkv, hd, True)
    (dx,) = torch.autograd.grad(o, x, do)
    dq, dkv = H * hd, Hkv * hd
    o2 = A.attention_tokens(x[:, :dq], x[:, dq:dq + dkv], x[:, dq + dkv:], B, S, S, H, Hkv, hd, True)
    (dx2,) = torch.autograd.grad(o2, x, do)
    assert torch.equal(o, o2) and torch.equal(dx, dx2)
    with torch.no_grad():
        assert torch.equal(A.attention_packed(x, B, S, H, Hkv, hd, True), o)


def test_non_finite_scores_behave_as_softmax_does():
    q = torch.ones(1, 1, 40, 16, device="cuda")
    k, v = torch.randn(1, 1, 40, 16, device="cuda"), torch.randn(1, 1, 40, 16, device="cuda")
    k[0, 0, 3] = float("-inf")
    k[0, 0, 20] = float("nan")
    o = A.attention_bhsd(q, k, v, True, None, 0)
    ref = _exact(q, k, v, True, 0)
    assert torch.equal(o.isnan(), ref.isnan())
    assert torch.allclose(o[~ref.isnan()], ref[~ref.isnan()], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("Sq,Sk,causal", [(1, 2, True), (1, 65, True), (1, 700, True), (4, 130, False), (40, 130, False)])
@pytest.mark.parametrize("H,Hkv,hd", [(2, 1, 64), (2, 2, 24)])
@pytest.mark.parametrize("what", ["value inf", "value -inf", "value nan", "key nan", "key inf", "scores -inf", "most scores -inf"])
@pytest.mark.parametrize("at", [0, -1, "middle"])
def test_non_finite_operands(Sq, Sk, causal, H, Hkv, hd, what, at):
    """Every key that these queries see, in the split form and in the tiles."""
    g = torch.Generator(device="cuda").manual_seed(Sk)
    q, k, v = (torch.randn(1, h, s, hd, device="cuda", generator=g) for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    q[..., 3] = 1.0
    j = Sk // 2 if at == "middle" else at
    kind, x = what.rsplit(" ", 1)
    if kind == "value":
        v[:, :, j, 5] = float(x)
    elif kind == "key":
        k[:, :, j, 3] = float(x)
    elif kind == "scores":
        k[:, :, j, 3] = float("-inf")
    else:
        keep = k[:, :, j].clone()
        k[..., 3] = float("-inf")
        k[:, :, j] = keep
    o = A.attention_bhsd(q, k, v, causal, None, Sk - Sq)
    d = [t.double() for t in (q, k, v)]
    s = d[0] @ d[1].repeat_interleave(H // Hkv, 1).transpose(-1, -2) / math.sqrt(hd)
    ref = s.softmax(-1) @ d[2].repeat_interleave(H // Hkv, 1)
    assert torch.equal(o.isnan(), ref.isnan()) and torch.equal(o.isinf(), ref.isinf())
    fin = ref.isfinite()
    assert torch.equal(o[ref.isinf()].double(), ref[ref.isinf()]) and torch.allclose(o[fin].double(), ref[fin], rtol=1e-5, atol=1e-5)


# Row tiles whose keys several CTAs divide: four (few rows; the first causal rows leave some without a key tile) and two (as many
# rows as the chip has SMs), the fewest tiles that are divided, ragged ends, offsets and odd head sizes.  The bound is that above: the
# parts meet in at most four more products and sums.
@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,hd,causal,off", [
    (1, 2, 2, 193, 193, 64, True, 0), (1, 2, 1, 257, 257, 32, False, 0), (2, 3, 3, 64, 450, 10, True, 386), (1, 1, 1, 33, 511, 128, False, 0),
    (1, 12, 12, 481, 481, 64, True, 0), (1, 10, 5, 509, 513, 64, False, 0), (1, 6, 2, 1000, 1000, 128, True, 0), (1, 16, 16, 449, 449, 16, True, 0)])
@pytest.mark.parametrize("what", ["finite", "value inf", "value -inf", "key nan", "scores -inf", "most scores -inf"])
def test_rows_with_shared_keys(B, H, Hkv, Sq, Sk, hd, causal, off, what):
    g = torch.Generator(device="cuda").manual_seed(Sk)
    q, k, v = (torch.randn(B, h, s, hd, device="cuda", generator=g) for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    q[..., 3] = 1.0
    kind, _, x = what.rpartition(" ")
    if kind == "value":
        v[:, :, Sk // 2, 5] = float(x)
    elif kind == "key":
        k[:, :, Sk // 2, 3] = float(x)
    elif kind == "scores":
        k[:, :, 0, 3] = float("-inf")
    elif kind:
        k[:, :, 70:, 3] = float("-inf")
    o = A.attention_bhsd(q, k, v, causal, None, off)
    ref = _exact(q.double(), k.double(), v.double(), causal, off)
    if kind == "value":      # a weight of zero times the value: rows that do not see the key are exact without it
        i = torch.arange(Sq, device="cuda") + off
        seen = i >= Sk // 2 if causal else torch.ones_like(i, dtype=torch.bool)
        v[:, :, Sk // 2, 5] = 0.0
        ref = _exact(q.double(), k.double(), v.double(), causal, off)
        assert torch.equal(o[:, :, seen, 5], torch.full_like(o[:, :, seen, 5], float(x)))
        o, ref = o.clone(), ref.clone()
        o[..., 5] = ref[..., 5].float()
    assert torch.equal(o.isnan(), ref.isnan())
    fin = ref.isfinite()
    assert float((o.double() - ref)[fin].norm()) <= 3e-6 * float(ref[fin].norm())
    if what == "finite":
        a = [t.requires_grad_(True) for t in (q, k, v)]
        d = [t.detach().double().requires_grad_(True) for t in a]
        do = torch.randn(o.shape, device="cuda", generator=g)
        got = torch.autograd.grad(A.attention_bhsd(*a, causal, None, off), a, do)
        for x, y in zip(got, torch.autograd.grad(_exact(*d, causal, off), d, do.double())):
            assert float((x.double() - y).norm() / y.norm()) < 3e-6
