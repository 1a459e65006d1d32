"""The native stack call against the modules' own forward passes: the same kernels, so the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import dart_pytorch_b200 as dp
from dart_pytorch_b200.models.bert import BertConfig, BertModel
from dart_pytorch_b200.models.llama import Llama, LlamaConfig
from dart_pytorch_b200.models.vit import ViTClassifier
from dart_pytorch_b200.nn.attention import EncoderCache
from dart_pytorch_b200.nn.transformer import Activation
from dart_pytorch_b200.ops import stack

DTYPES = [torch.bfloat16, torch.float32]


def _both(monkeypatch, fn):
    """``fn()`` through the native call (which has to have run) and through the modules."""
    calls, run = [], stack.run

    def counted(*a, **k):
        out = run(*a, **k)
        calls.append(out is not None)
        return out
    with torch.no_grad():
        monkeypatch.setattr(stack, "run", counted)
        native = fn()
        assert calls and all(calls)
        monkeypatch.setattr(stack, "run", lambda *a, **k: None)
        plain = fn()
        monkeypatch.setattr(stack, "run", run)
    return native, plain


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert x.shape == y.shape and x.dtype == y.dtype and torch.equal(x, y)


def _gpt(dtype, layers, heads, hd, act=Activation.geluTanh, bias=True):
    return dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=300, embed_dim=heads * hd, num_layers=layers, num_heads=heads,
                               attn_bias=bias, activation=act, device="cuda", dtype=dtype, init_std=0.05)).eval()


def _steps(model, cache, toks, n):
    out = [model.hidden(toks[..., :n], 0, cache)]
    for i in range(n, toks.shape[-1]):
        out.append(model.hidden(toks[..., i:i + 1], i, cache))
    return out + [c.k_buf for c in cache.layers] + [c.v_buf for c in cache.layers]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("layers", [1, 2, 3])
@pytest.mark.parametrize("shape,n", [((7,), 4), ((1, 1), 1), ((3, 40), 37), ((70, 3), 1)])
def test_gpt(monkeypatch, dtype, layers, shape, n):
    m = _gpt(dtype, layers, 2, 64, act=[Activation.geluTanh, Activation.relu, Activation.quickGelu][layers - 1], bias=layers != 2)
    toks = torch.randint(0, 97, shape, device="cuda")
    _same(*_both(monkeypatch, lambda: [m.hidden(toks)]))
    _same(*_both(monkeypatch, lambda: _steps(m, EncoderCache.empty(layers, 2, max_len=60), toks, n)))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,Hkv,hd", [(4, 1, 64), (4, 2, 128), (4, 2, 32)])
@pytest.mark.parametrize("shape,n", [((9,), 8), ((33, 20), 18)])
def test_llama(monkeypatch, dtype, H, Hkv, hd, shape, n):
    m = Llama(LlamaConfig(vocab_size=97, max_ctx=64, embed_dim=H * hd, num_layers=3, num_heads=H, num_kv_heads=Hkv, ffn_dim=200,
                          device="cuda", dtype=dtype, init_std=0.05)).eval()
    toks = torch.randint(0, 97, shape, device="cuda")
    _same(*_both(monkeypatch, lambda: [m.hidden(toks)]))
    _same(*_both(monkeypatch, lambda: _steps(m, m.new_cache(), toks, n)))


@pytest.mark.parametrize("dtype,hd", [(torch.bfloat16, 64), (torch.bfloat16, 32), (torch.bfloat16, 96), (torch.float32, 32), (torch.float32, 24)])
@pytest.mark.parametrize("shape", [(5,), (1, 23), (6, 33)])
def test_bert(monkeypatch, dtype, hd, shape):
    m = BertModel(BertConfig(vocab_size=97, max_position_embeddings=64, embed_dim=4 * hd, num_layers=3, num_heads=4,
                             intermediate_size=136, device="cuda", dtype=dtype)).eval()
    toks = torch.randint(0, 97, shape, device="cuda")
    _same(*_both(monkeypatch, lambda: [m(toks)]))


@pytest.mark.parametrize("dtype", DTYPES)
def test_vit(monkeypatch, dtype):
    m = ViTClassifier(image_size=32, patch_size=8, embed_dim=128, num_layers=2, num_heads=2, num_classes=7, device="cuda",
                      dtype=dtype).eval()
    x = torch.randn(3, 3, 32, 32, device="cuda").to(dtype)
    _same(*_both(monkeypatch, lambda: [m(x)]))


def test_declined(monkeypatch):
    """What the native call does not stand for keeps its own path, and its errors."""
    run, outs = stack.run, []
    monkeypatch.setattr(stack, "run", lambda *a, **k: (outs.append(run(*a, **k)), outs[-1])[1])
    m, toks = _gpt(torch.float32, 2, 2, 64), torch.randint(0, 97, (2, 5), device="cuda")
    assert m.hidden(toks).requires_grad and not outs                      # gradients
    with torch.no_grad():
        want = m.hidden(toks)
        assert outs.pop() is not None
        half = EncoderCache.empty(2, 2)
        m.hidden(toks, 0, half)
        outs.clear()
        half.layers[1].seq_len = 4                                        # layers of different lengths
        m.hidden(toks[:, :1], 5, half)
        assert not [o for o in outs if o is not None]
        outs.clear()
        with pytest.raises(ValueError):                                   # another batch than the cache's
            m.hidden(toks[:1], 0, half)
        m.encoder.blocks[0].ffn1.forward = lambda *a, **k: None           # a replaced module
        outs.clear()
        m.hidden(toks)
        assert not outs
        del m.encoder.blocks[0].ffn1.__dict__["forward"]
        m.train()
        m.encoder.blocks[1].dropout.p = 0.5                               # dropout in training
        m.hidden(toks)
        assert not outs
        m.eval()
        assert torch.equal(m.hidden(toks), want) and outs.pop() is not None
        assert torch.equal(m.hidden(toks.int()), want)                    # other token types: looked up by the module
        assert [o is None for o in outs] == [True, False]
