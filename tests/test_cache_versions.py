"""Kernels that write a cache in place count as in-place operations: a graph that saved its buffers is refused afterwards."""
import pytest
import torch

import dart_pytorch_b200 as dp
from dart_pytorch_b200.nn.attention import EncoderCache, MHACache, MultiHeadAttention
from dart_pytorch_b200.ops import decode


def _saved(cache):
    w = torch.ones_like(cache.k_buf).requires_grad_(True)
    return [(buf * w).sum() for buf in (cache.k_buf, cache.v_buf)]


def _refused(sums):
    for y in sums:
        with pytest.raises(RuntimeError, match="inplace"):
            y.backward()


def test_rows_of_a_projection(monkeypatch):
    monkeypatch.setattr(decode, "rows_to_cache", lambda *a: None)
    cache = MHACache(2, 16)
    cache.append(torch.randn(1, 3, 8), torch.randn(1, 3, 8))
    sums = _saved(cache)
    cache.append_rows(torch.randn(2, 24), 1, 2, 2, 2, 4)
    _refused(sums)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("native", [True, False])
def test_steps_of_a_model(dtype, native):
    if native:
        m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=64, embed_dim=128, num_layers=2, num_heads=2, device="cuda", dtype=dtype)).eval()
        cache = EncoderCache.empty(2, 2)
        step = lambda pos: m.hidden(torch.zeros(2, 3, dtype=torch.long, device="cuda"), pos, cache)     # noqa: E731
        layer = cache.layers[1]
    else:
        att, layer = MultiHeadAttention(128, 2, device="cuda", dtype=dtype), MHACache(2)
        step = lambda pos: att(torch.zeros(2, 3, 128, device="cuda", dtype=dtype), cache=layer, causal=True)     # noqa: E731
    with torch.no_grad():
        step(0)
    sums = _saved(layer)
    with torch.no_grad():
        step(3)
    _refused(sums)
