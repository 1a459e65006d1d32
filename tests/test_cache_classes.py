"""Key / value caches of the caller's own: whatever has ``append`` and ``seq_len`` is asked for its rows."""
import pytest
import torch

import dart_pytorch_b200 as dp
from dart_pytorch_b200.nn.attention import EncoderCache, MHACache, MultiHeadAttention


class Appending:
    """Nothing but ``append`` and ``seq_len``.  ``gap``: elements between the rows it hands over, ``skip``: between its sequences."""

    def __init__(self, gap=0, skip=0):
        self.seq_len, self.kept, self.gap, self.skip, self.calls = 0, [], gap, skip, 0

    def _rows(self, ts):
        t = torch.cat(ts, 1)
        B, n, w = t.shape
        room = torch.zeros(B, n * (w + self.gap) + self.skip, dtype=t.dtype, device=t.device)
        rows = room.as_strided((B, n, w), (room.stride(0), w + self.gap, 1))
        rows.copy_(t)
        return rows

    def append(self, k_new, v_new):
        self.calls += 1
        self.kept.append((k_new, v_new))
        self.seq_len += k_new.shape[1]
        return self._rows([k for k, _ in self.kept]), self._rows([v for _, v in self.kept])


class Halving(MHACache):
    """Keeps half of every key: a stand-in for caches that store something else than they are given."""

    def append(self, k_new, v_new):
        return super().append(k_new * 0.5, v_new)


def _steps(att, x, cache, n):
    with torch.no_grad():
        out = [att(x[:, :n], cache=cache, causal=True)]
        for i in range(n, x.shape[1]):
            out.append(att(x[:, i:i + 1], cache=cache, start_pos=i))
    return torch.cat(out, 1)


def test_a_cache_with_nothing_but_append():
    att, x, cache = MultiHeadAttention(32, 4), torch.randn(2, 7, 32), Appending()
    got = _steps(att, x, cache, 4)
    with torch.no_grad():
        assert torch.allclose(got, att(x, causal=True), atol=1e-6)
    assert cache.calls == 4 and cache.seq_len == 7


@pytest.mark.parametrize("how", ["subclass", "object"])
def test_the_callers_append_is_not_passed_by(monkeypatch, how):
    """As on a device, where the stock cache takes rows straight from the projection."""
    monkeypatch.setattr(MHACache, "takes_rows", lambda self, qkv: True)
    monkeypatch.setattr(MHACache, "append_rows", None)
    seen = []
    cache = Halving(4) if how == "subclass" else MHACache(4)
    if how == "object":
        cache.append = lambda k, v: (seen.append(1), MHACache.append(cache, k, v))[1]
    _steps(MultiHeadAttention(32, 4), torch.randn(2, 5, 32), cache, 4)
    assert cache.seq_len == 5 and (how == "subclass" or len(seen) == 2)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hd", [64, 32])
def test_models_append_through_the_callers_cache(dtype, hd):
    m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=64, embed_dim=2 * hd, num_layers=2, num_heads=2, attn_bias=True, device="cuda",
                            dtype=dtype, init_std=0.2)).eval()
    toks = torch.randint(0, 97, (2, 9), device="cuda")

    def steps(cache):
        with torch.no_grad():
            return torch.cat([m.hidden(toks[:, :7], 0, cache)] + [m.hidden(toks[:, i:i + 1], i, cache) for i in (7, 8)], 1)
    stock = EncoderCache.empty(2, 2)
    want = steps(stock)
    own = EncoderCache([Appending(), Appending()])
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-5      # the same sums in another order: a few roundings a layer
    assert float((steps(own) - want).float().norm() / want.float().norm()) < tol
    assert [c.calls for c in own.layers] == [3, 3]
    half = EncoderCache([Halving(2), Halving(2)])
    steps(half)
    first = half.layers[0]
    assert torch.equal(first.k_buf[:, :9], stock.layers[0].k_buf[:, :9] * 0.5)
    assert torch.equal(first.v_buf[:, :9], stock.layers[0].v_buf[:, :9])


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [24, 32, 96])
@pytest.mark.parametrize("gap,skip", [(0, 0), (8, 0), (0, 8), (1, 0), (0, 1)])
def test_rows_in_any_layout(hd, gap, skip):
    """Heads that are no kernel size of their own, on rows that start anywhere and sequences that are any distance apart."""
    att = MultiHeadAttention(4 * hd, 4, num_kv_heads=2, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(3, 9, 4 * hd, device="cuda", dtype=torch.bfloat16)
    got = _steps(att, x, Appending(gap, skip), 6)
    with torch.no_grad():
        want = att(x, causal=True)
    assert float((got - want).float().norm() / want.float().norm()) < 1e-2
