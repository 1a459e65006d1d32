"""Steps through the native stack (a chain of dependent launches, the cache append inside the attention) against the modules' own
forward passes: the same bits, in the hidden states and in the caches."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import dart_pytorch_b200 as dp
from dart_pytorch_b200.models.llama import Llama, LlamaConfig
from dart_pytorch_b200.nn.attention import EncoderCache
from dart_pytorch_b200.nn.transformer import Activation
from dart_pytorch_b200.ops import stack


def _steps(model, cache, toks, n):
    with torch.no_grad():
        out = [model.hidden(toks[:, :n], 0, cache)]
        for i in range(n, toks.shape[1]):
            out.append(model.hidden(toks[:, i:i + 1], i, cache))
    return out + [c.k_buf for c in cache.layers] + [c.v_buf for c in cache.layers]


def _both(monkeypatch, fn):
    native = fn()
    with monkeypatch.context() as m:
        m.setattr(stack, "run", lambda *a, **k: None)
        plain = fn()
    for x, y in zip(native, plain, strict=True):
        assert torch.equal(x, y)


# rows up to 8 stream the weights and from 256 terms on take the norm with them (9 rows and 1032 columns do not); tokens go past a tile
# of 64 keys, and 3 at a time into it
@pytest.mark.parametrize("width,heads", [(256, 4), (264, 3), (1024, 8), (1032, 12)])
@pytest.mark.parametrize("B,n", [(1, 62), (3, 1), (8, 126), (9, 3)])
def test_gpt(monkeypatch, width, heads, B, n):
    m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=300, embed_dim=width, num_layers=2, num_heads=heads, ffn_dim=300, attn_bias=True,
                            activation=Activation.geluTanh, device="cuda", dtype=torch.float32, init_std=0.05)).eval()
    toks = torch.randint(0, 97, (B, n + 4), device="cuda")
    _both(monkeypatch, lambda: _steps(m, EncoderCache.empty(2, heads, max_len=300), toks, n))


@pytest.mark.parametrize("B,n,S", [(1, 63, 3), (2, 5, 4), (1, 0, 2)])
def test_several_tokens_a_step(monkeypatch, B, n, S):
    m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=300, embed_dim=256, num_layers=2, num_heads=4, ffn_dim=300, attn_bias=False,
                            activation=Activation.relu, device="cuda", dtype=torch.float32, init_std=0.05)).eval()
    toks = torch.randint(0, 97, (B, n + S), device="cuda")

    def run():
        cache = EncoderCache.empty(2, 4, max_len=300)
        with torch.no_grad():
            out = [m.hidden(toks[:, :n], 0, cache)] if n else []
            out.append(m.hidden(toks[:, n:], n, cache))
        return out + [c.k_buf for c in cache.layers] + [c.v_buf for c in cache.layers]
    _both(monkeypatch, run)


@pytest.mark.parametrize("B", [1, 8, 9])
def test_llama(monkeypatch, B):
    m = Llama(LlamaConfig(vocab_size=97, max_ctx=300, embed_dim=512, num_layers=2, num_heads=8, num_kv_heads=2, ffn_dim=264,
                          device="cuda", dtype=torch.float32, init_std=0.05)).eval()
    toks = torch.randint(0, 97, (B, 68), device="cuda")
    _both(monkeypatch, lambda: _steps(m, m.new_cache(), toks, 62))


# Both ends of the chained steps; every repetition gives the same bits.
@pytest.mark.parametrize("width,heads", [(128, 2), (512, 8), (1024, 16)])
@pytest.mark.parametrize("B,n", [(1, 24), (33, 1), (1, 64), (5, 13), (128, 1), (1, 129), (2, 128), (257, 1)])
def test_chained_steps(monkeypatch, width, heads, B, n):
    m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=300, embed_dim=width, num_layers=3, num_heads=heads, ffn_dim=4 * width, attn_bias=True,
                            activation=Activation.geluTanh, device="cuda", dtype=torch.float32, init_std=0.05)).eval()
    toks = torch.randint(0, 97, (B, n + 2), device="cuda")
    run = lambda: _steps(m, EncoderCache.empty(3, heads, max_len=300), toks, n)
    _both(monkeypatch, run)
    first = run()
    for _ in range(10):
        assert all(torch.equal(x, y) for x, y in zip(first, run()))


# bf16 prompts on both sides of the longest chain (12 M activations): tiled products and attention as dependents, several query tiles and
# two heads a CTA.
@pytest.mark.parametrize("width,heads,B,n", [(384, 12, 8, 119), (384, 6, 1, 300), (768, 12, 3, 65), (1024, 16, 16, 128), (2048, 16, 47, 128)])
def test_chained_bf16_prompts(monkeypatch, width, heads, B, n):
    m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=300, embed_dim=width, num_layers=3, num_heads=heads, ffn_dim=2 * width, attn_bias=True,
                            activation=Activation.geluTanh, device="cuda", dtype=torch.bfloat16, init_std=0.05)).eval()
    toks = torch.randint(0, 97, (B, n), device="cuda")

    def run():
        with torch.no_grad():
            return [m.hidden(toks)]
    _both(monkeypatch, run)
    first = run()
    for _ in range(10):
        assert torch.equal(first[0], run()[0])


def test_infinities_and_nan(monkeypatch):
    m = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=300, embed_dim=256, num_layers=1, num_heads=4, ffn_dim=300, attn_bias=True,
                            activation=Activation.relu, device="cuda", dtype=torch.float32, init_std=0.05)).eval()
    toks = torch.randint(0, 97, (3, 6), device="cuda")
    with torch.no_grad():
        table = m.parameters()[0].data
        table[toks[0, 5], 3], table[toks[1, 5], 4] = float("inf"), float("nan")
    def run():
        return [t.nan_to_num(1.5) for t in _steps(m, EncoderCache.empty(1, 4, max_len=300), toks, 5)]
    _both(monkeypatch, run)
