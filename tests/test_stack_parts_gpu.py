"""Models whose parts have been replaced keep the parts that were put in: the native stack call does not go past them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import dart_pytorch_b200 as dp
from dart_pytorch_b200.models.bert import BertConfig, BertModel
from dart_pytorch_b200.models.llama import Llama, LlamaConfig
from dart_pytorch_b200.nn.attention import EncoderCache, RopeCache
from dart_pytorch_b200.nn.module import Module
from dart_pytorch_b200.nn.transformer import Activation


class Around(Module):
    """Another module in the place of one, with nothing of it but its call."""

    def __init__(self, inner, seen):
        super().__init__()
        self.inner, self.seen = inner, seen

    def submodules(self):
        return [self.inner]

    def forward(self, *a, **k):
        self.seen.append(1)
        return self.inner(*a, **k)


class StrictRope(RopeCache):
    def check_window(self, start_pos, n):
        self.seen.append(1)
        super().check_window(start_pos, n)


def _models():
    kw = dict(device="cuda", dtype=torch.float32)
    gpt = dp.GPT(dp.GPTConfig(vocab_size=97, max_ctx=64, embed_dim=64, num_layers=2, num_heads=2, attn_bias=True, dropout_p=0.1,
                              activation=Activation.geluTanh, init_std=0.05, **kw))
    llama = Llama(LlamaConfig(vocab_size=97, max_ctx=64, embed_dim=64, num_layers=2, num_heads=2, num_kv_heads=1, ffn_dim=72,
                              init_std=0.05, **kw))
    bert = BertModel(BertConfig(vocab_size=97, max_position_embeddings=64, embed_dim=64, num_layers=2, num_heads=2,
                                intermediate_size=136, **kw))
    return {"gpt": gpt.eval(), "llama": llama.eval(), "bert": bert.eval()}


# the object that holds the part, the part's name, and whether another module takes its place or a method of the object does
MODULES = [("gpt", "", "embed_drop"), ("gpt", "", "encoder"), ("gpt", "encoder.blocks", 0), ("gpt", "encoder.blocks", 1),
           ("gpt", "encoder.blocks.1", "mha"), ("gpt", "encoder.blocks.0.mha", "wo"), ("gpt", "encoder.blocks.0.mha", "attn_dropout"),
           ("gpt", "encoder", "final_norm"), ("llama", "blocks", 0), ("llama", "blocks.1", "attn"), ("llama", "blocks.0", "ffn"),
           ("llama", "blocks.1.ffn", "down"), ("llama", "", "final_norm"), ("bert", "", "embeddings"), ("bert", "layers", 1),
           ("bert", "layers.0", "attention"), ("bert", "layers.0", "output_ln"), ("bert", "embeddings", "layer_norm")]
METHODS = [("gpt", "encoder", "forward"), ("gpt", "embed_drop", "forward"), ("gpt", "encoder.blocks.1", "forward"),
           ("gpt", "encoder.blocks.0.ln1", "with_residual"), ("gpt", "encoder.blocks.0.mha", "_attend_tokens"),
           ("llama", "", "hidden_from_embeddings"), ("llama", "blocks.0.ffn_norm", "with_residual"),
           ("llama", "blocks.0.attn", "_rope_qk"), ("llama", "rope", "check_window"), ("bert", "layers.0", "forward")]


def _at(model, path):
    for name in filter(None, path.split(".")):
        model = model[int(name)] if name.isdigit() else getattr(model, name)
    return model


def _run(name, model, toks, cached):
    if name == "bert":
        return model(toks)
    return model.hidden(toks, 0, EncoderCache.empty(2, 2 if name == "gpt" else 1) if cached else None)


def _check(name, model, toks, seen, want):
    for cached in (False, True):
        del seen[:]
        assert torch.equal(_run(name, model, toks, cached), want) and seen


@pytest.mark.parametrize("name,path,part", MODULES)
def test_another_module(name, path, part):
    model, toks, seen = _models()[name], torch.randint(0, 97, (2, 9), device="cuda"), []
    with torch.no_grad():
        want = _run(name, model, toks, False)
        owner = _at(model, path)
        if isinstance(part, int):
            owner[part] = Around(owner[part], seen)
        else:
            setattr(owner, part, Around(getattr(owner, part), seen))
        if (name, path, part) == ("gpt", "", "encoder"):
            model.encoder.blocks = None      # (an encoder needs no blocks of its own)
        _check(name, model, toks, seen, want)


@pytest.mark.parametrize("name,path,method", METHODS)
def test_a_method_replaced_on_the_object(name, path, method):
    model, toks, seen = _models()[name], torch.randint(0, 97, (2, 9), device="cuda"), []
    with torch.no_grad():
        want = _run(name, model, toks, False)
        owner = _at(model, path)
        stock = getattr(owner, method)
        setattr(owner, method, lambda *a, **k: (seen.append(1), stock(*a, **k))[1])
        if method in ("_attend_tokens", "_rope_qk"):      # (each is called with, or without, a cache only)
            del seen[:]
            assert torch.equal(_run(name, model, toks, method == "_attend_tokens"), want) and seen
        else:
            _check(name, model, toks, seen, want)


def test_a_rope_class_of_the_callers_own():
    model, toks, seen = _models()["llama"], torch.randint(0, 97, (2, 9), device="cuda"), []
    with torch.no_grad():
        want = model.hidden(toks)
        rope = StrictRope(64, 32, base=model.rope.base)
        rope.seen = seen
        for b in model.blocks:
            b.attn.rope = rope
        _check("llama", model, toks, seen, want)


def test_an_embedding_dropout_without_a_rate_trains():
    model, toks, seen = _models()["gpt"], torch.randint(0, 97, (2, 9), device="cuda"), []
    model.embed_drop = Around(model.embed_drop, seen)
    model.train()
    assert model.hidden(toks).requires_grad and seen
