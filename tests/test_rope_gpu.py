"""Rotary embedding and its fusion with the cache append, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.nn.attention import MHACache, MultiHeadAttention, RopeCache
from dart_pytorch_b200.ops import decode as D
from dart_pytorch_b200.ops import kernels as K

# bf16 results are rounded once from fp32 (half a unit of 2^-8 of the value); fp32 angles of up to `pos` radians carry
# an error of about pos * 2^-23 into the sine and cosine.
TOL = {torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -20}


def _turn(x, heads, hd, rot, pos, base, inverse=False):
    """``x [tokens, heads * hd]`` in fp64 at integer positions ``pos [tokens]``."""
    x = x.double().reshape(-1, heads, hd).clone()
    half = rot // 2
    if half:
        ang = pos.double().view(-1, 1, 1) * base ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / rot)
        a, b = x[..., :half].clone(), x[..., half:rot].clone()
        s = -ang.sin() if inverse else ang.sin()
        x[..., :half], x[..., half:rot] = a * ang.cos() - b * s, b * ang.cos() + a * s
    return x.reshape(-1, heads * hd)


def _close(got, want, dtype, pos_max):
    tol = max(TOL[dtype], pos_max * 2.0 ** -22)
    assert float((got.double() - want).abs().max()) <= tol * float(want.abs().max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,heads,hd,rot,pad", [(1, 1, 2, 2, 0), (7, 3, 20, 12, 1), (33, 5, 64, 64, 8), (900, 4, 128, 128, 0),
                                                     (5000, 2, 64, 16, 0), (9, 1, 1200, 1100, 0),
                                                     (5000, 1, 1200, 1100, 0)])
@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("seq_len,start", [(0, 3), (4, 11)])
def test_rope(dtype, tokens, heads, hd, rot, pad, inverse, seq_len, start):
    x = torch.randn(tokens, heads * hd + pad, device="cuda").to(dtype)
    t = torch.arange(tokens, device="cuda")
    pos = start + (t % seq_len if seq_len else t)
    want = _turn(x[:, :heads * hd], heads, hd, rot, pos, 10000.0, inverse)
    out = torch.full((tokens, heads * hd), 7.0, device="cuda").to(dtype)
    K.rope(x, heads, hd, rot, seq_len, start, 10000.0, inverse=inverse, out=out)
    _close(out, want, dtype, start + tokens)
    behind = x[:, heads * hd:].clone()
    K.rope(x, heads, hd, rot, seq_len, start, 10000.0, inverse=inverse)
    assert torch.equal(x[:, :heads * hd], out) and torch.equal(x[:, heads * hd:], behind)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,Hkv,hd,rot", [(4, 2, 64, 64), (3, 1, 20, 8), (2, 2, 32, 0), (6, 3, 128, 96)])
@pytest.mark.parametrize("B,S,pos0,row0", [(1, 1, 9, 9), (3, 5, 4, 17), (2, 700, 0, 1)])
def test_rows_to_cache(dtype, H, Hkv, hd, rot, B, S, pos0, row0):
    qkv = torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda").to(dtype)
    kc, vc = (torch.full((B, row0 + S + 3, Hkv * hd), 5.0, device="cuda").to(dtype) for _ in range(2))
    pos = pos0 + torch.arange(S, device="cuda").repeat(B)
    want = _turn(qkv[:, :(H + Hkv) * hd], H + Hkv, hd, rot, pos, 10000.0)
    v, before = qkv[:, (H + Hkv) * hd:].clone(), qkv.clone()
    D.rows_to_cache(qkv, kc, vc, B, S, H, Hkv, hd, pos0, row0, rot)
    _close(qkv[:, :H * hd], want[:, :H * hd], dtype, pos0 + S)
    assert torch.equal(qkv[:, H * hd:], before[:, H * hd:])
    _close(kc[:, row0:row0 + S].reshape(B * S, -1), want[:, H * hd:], dtype, pos0 + S)
    assert torch.equal(vc[:, row0:row0 + S].reshape(B * S, -1), v)
    for c in (kc, vc):
        assert (c[:, :row0] == 5.0).all() and (c[:, row0 + S:] == 5.0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,Hkv,hd,rope", [(4, 1, 64, True), (8, 8, 128, False), (2, 2, 32, True), (16, 1, 64, True)])
def test_cached_steps_equal_one_pass(dtype, H, Hkv, hd, rope):
    D_, n = H * hd, 150
    r = RopeCache(256, hd, base=10000.0) if rope else None
    att = MultiHeadAttention(D_, H, num_kv_heads=Hkv, bias=True, device="cuda", dtype=dtype, rope=r, seed=3)
    x = torch.randn(2, n, D_, device="cuda").to(dtype)
    with torch.no_grad():
        want = att(x, causal=True)
        cache = MHACache(Hkv, 256)
        got = [att(x[:, :140], cache=cache, causal=True)]
        for i in range(140, n):
            got.append(att(x[:, i:i + 1], cache=cache, start_pos=i))
    got = torch.cat(got, 1)
    assert cache.seq_len == n
    # the same sums in another order: a few units of the dtype's rounding
    assert float((got - want).float().norm() / want.float().norm()) < (1e-2 if dtype == torch.bfloat16 else 2e-6)
