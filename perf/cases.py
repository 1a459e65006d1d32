"""Performance cases: what programs built on this package spend their GPU time on, through its public entry points.

Four kinds of work, over the dense families (GPT, Llama, ViT, BERT) and both dtypes the models run in:

* ``train``: one ``Trainer.step`` (loss, backward, clipping at 1.0, AdamW) of a run resumed at step 1000;
* ``prompt``: the prompt pass of generation: a new key / value cache, the hidden states of the prompts, the logits after
  each prompt's last token;
* ``decode``: one token more for every sequence after such a prompt pass;
* ``encode``: the token features of a batch of texts.

bfloat16 is what training and serving at size run in; float32 is the default dtype of every configuration class and of the
command-line trainers and runners.  Each case carries its own sizes as plain values; weights and inputs are made from a
seed alone and ``exact`` computes the same pass in float64 with plain torch.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as TF
from torch.utils.checkpoint import checkpoint

import dart_pytorch_b200 as dp
from dart_pytorch_b200 import ops
from dart_pytorch_b200.models.bert import BertConfig, BertModel
from dart_pytorch_b200.models.llama import Llama, LlamaConfig
from dart_pytorch_b200.models.vit import ViTClassifier
from dart_pytorch_b200.nn.attention import EncoderCache
from dart_pytorch_b200.nn.transformer import Activation
from dart_pytorch_b200.utils.trainer import Trainer

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
INIT_STD = 0.02
ROPE_BASE = 500000.0
LR, BETA1, BETA2, EPS, DECAY, CLIP, RESUMED = 6e-5, 0.9, 0.95, 1e-8, 0.1, 1.0, 1000
ARENA_ALIGN = 128      # elements every parameter of an optimizer's flat range is padded to


def _case(name, kind, family, dtype, batch, seq, dim, layers, heads, kv_heads, ffn, vocab, image=0, patch=0):
    c = dict(kind=kind, family=family, dtype=dtype, batch=batch, seq=seq, dim=dim, layers=layers, heads=heads,
             kv_heads=kv_heads, ffn=ffn, vocab=vocab, image=image, patch=patch)
    return {"name": name, **c} if name else c


def listed():
    return [
        # the headline benchmark's workload: GPT-2 124M, 16 sequences of 1024 tokens
        _case("train_gpt2_124m", "train", "gpt", "bf16", 16, 1024, 768, 12, 12, 12, 3072, 50257),
        # ViT-B/16 on 224 x 224 images, batch 128: 197 tokens a sequence, not causal
        _case("train_vit_b16", "train", "vit", "bf16", 128, 197, 768, 12, 12, 12, 3072, 1000, 224, 16),
        # a Llama-shaped model with grouped queries and heads of 64; an odd context, as packed documents leave it
        _case("train_llama_1024", "train", "llama", "bf16", 4, 1531, 1024, 6, 16, 4, 2816, 32768),
        # the smallest training that uses the kernels in earnest: a step is a chain of short launches
        _case("train_gpt_small", "train", "gpt", "bf16", 3, 201, 128, 2, 2, 2, 512, 320),
        # the command line's larger character-level trainer (its default dtype, batch and context)
        _case("train_gpt_char_fp32", "train", "gpt", "fp32", 8, 128, 256, 6, 8, 8, 1024, 65),
        # prompts of a served Llama-shaped model, heads of 128
        _case("prompt_llama_2048", "prompt", "llama", "bf16", 4, 2048, 2048, 6, 16, 4, 5504, 32768),
        # the same model while it generates for 32 users
        _case("decode_llama_2048", "decode", "llama", "bf16", 32, 2048, 2048, 6, 16, 4, 5504, 32768),
        # GPT-2 124M as the runners load it by default, a prompt of odd length ...
        _case("prompt_gpt2_fp32", "prompt", "gpt", "fp32", 1, 509, 768, 12, 12, 12, 3072, 50257),
        # ... and its tokens after that
        _case("decode_gpt2_fp32", "decode", "gpt", "fp32", 1, 509, 768, 12, 12, 12, 3072, 50257),
        # sentence embeddings (a MiniLM-sized BERT, heads of 32): a batch while an index is built, one query while it is
        # searched
        _case("encode_bert_batch", "encode", "bert", "bf16", 64, 119, 384, 6, 12, 12, 1536, 30522),
        _case("encode_bert_query_fp32", "encode", "bert", "fp32", 1, 23, 384, 6, 12, 12, 1536, 30522),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind, family, dtype = rng.choice([
        ("train", "gpt", "bf16"), ("train", "gpt", "bf16"), ("train", "llama", "bf16"), ("train", "vit", "bf16"),
        ("train", "gpt", "fp32"), ("prompt", "llama", "bf16"), ("prompt", "gpt", "bf16"), ("prompt", "gpt", "fp32"),
        ("decode", "llama", "bf16"), ("decode", "gpt", "fp32"), ("encode", "bert", "bf16"), ("encode", "bert", "fp32")])
    half = dtype == "bf16"
    head = rng.choice([64, 64, 128]) if family == "llama" and kind != "train" else \
        rng.choice([64, 64, 32]) if half else rng.choice([16, 32, 64])
    heads = _spread(rng, 2, (2048 if head == 128 else 1024) // head if half else 768 // head)
    kv = heads
    if family == "llama":
        heads = max(4, heads // 4 * 4)
        kv = heads // 4
    dim = heads * head
    layers = rng.randint(1, 6)
    ffn = (dim * 11 // 4 + 7) // 8 * 8 if family == "llama" else 4 * dim
    vocab = _spread(rng, 65, 50257)
    image = patch = 0
    if family == "vit":
        patch = rng.choice([8, 16])
        image = patch * rng.randint(4, 14)
        seq, batch, vocab = (image // patch) ** 2 + 1, _spread(rng, 4, 128), rng.randint(2, 1000)
    elif kind == "train":
        seq = _spread(rng, 64, 1024) if half else _spread(rng, 32, 256)
        batch = _spread(rng, 1, max(1, 8192 // seq)) if half else _spread(rng, 1, 8)
        if not half:
            layers = max(1, min(layers, 384 // (batch * heads)))
    elif kind == "encode":
        seq, batch = _spread(rng, 8, 512), _spread(rng, 1, 64) if half else rng.randint(1, 2)
    else:
        seq = _spread(rng, 64, 2048) if half else _spread(rng, 16, 1024)
        batch = _spread(rng, 1, 32 if kind == "decode" else max(1, 8192 // seq)) if half else 1
    return _case(None, kind, family, dtype, batch, seq, dim, layers, heads, kv, ffn, vocab, image, patch)


# ------------------------------------------------------------------------------------------------ weights and inputs
def _parameters(c):
    """``[(name, shape, mean)]`` in the models' own parameter order."""
    D, H, Hkv, F, V = c["dim"], c["heads"], c["kv_heads"], c["ffn"], c["vocab"]
    hd = D // H
    fam = c["family"]
    out = []

    def norm(name):
        out.append((name + ".g", (D,), 1.0))
        if fam != "llama":
            out.append((name + ".b", (D,), 0.0))

    def linear(name, n, k, bias=True):
        out.append((name + ".w", (n, k), 0.0))
        if bias:
            out.append((name + ".b", (n,), 0.0))
    if fam in ("gpt", "llama"):
        out.append(("tok", (V, D), 0.0))
        if fam == "gpt":
            out.append(("pos", (c["seq"] + 128, D), 0.0))
    elif fam == "bert":
        out += [("tok", (V, D), 0.0), ("pos", (c["seq"], D), 0.0), ("type", (1, D), 0.0)]
        norm("ln0")
    else:
        linear("patch", D, 3 * c["patch"] ** 2)
        out += [("cls", (1, D), 0.0), ("pos", (c["seq"], D), 0.0)]
    for i in range(c["layers"]):
        p = f"{i}."
        bias = fam != "llama"
        if fam != "bert":
            norm(p + "n1")
            norm(p + "n2")
        linear(p + "qkv", (H + 2 * Hkv) * hd, D, bias)
        linear(p + "wo", D, H * hd, bias)
        if fam == "bert":
            norm(p + "n1")
        if fam == "llama":
            linear(p + "gu", 2 * F, D, False)
        else:
            linear(p + "f1", F, D)
        linear(p + "f2", D, F, bias)
        if fam == "bert":
            norm(p + "n2")
    if fam != "bert":
        norm("lnf")
    if fam == "vit":
        linear("head", V, D)
    return out


def _weights(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[c["dtype"]]
    return {n: (torch.randn(s, generator=g, device="cuda") * INIT_STD + mean).to(dt) for n, s, mean in _parameters(c)}


def _inputs(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 77777)
    B, S, V = c["batch"], c["seq"], c["vocab"]
    if c["family"] == "vit":
        images = torch.randn(B, 3, c["image"], c["image"], generator=g, device="cuda").to(DTYPES[c["dtype"]])
        return images, torch.randint(0, V, (B,), generator=g, device="cuda")
    tokens = torch.randint(0, V, (B, S + 1), generator=g, device="cuda")
    return tokens[:, :-1].contiguous(), tokens[:, 1:].contiguous()


def _moments(numel, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 55555)
    m = torch.randn(numel, generator=g, device="cuda") * 1e-4
    v = (torch.rand(numel, generator=g, device="cuda") + 0.5) * 1e-7
    return m, v


def _arena(c, values, dtype):
    """Parameters in the layout of an optimizer's flat range: last one first, each padded."""
    parts = []
    for n, s, _ in reversed(_parameters(c)):
        k = math.prod(s)
        parts.append(values[n].reshape(-1).to(dtype))
        pad = -k % ARENA_ALIGN
        if pad:
            parts.append(torch.zeros(pad, dtype=dtype, device="cuda"))
    return torch.cat(parts)


def _model(c, weights):
    dt = DTYPES[c["dtype"]]
    D, L, H, F, V = c["dim"], c["layers"], c["heads"], c["ffn"], c["vocab"]
    fam = c["family"]
    kw = dict(device="cuda", dtype=dt)
    if fam == "gpt":
        m = dp.GPT(dp.GPTConfig(vocab_size=V, max_ctx=c["seq"] + 128, embed_dim=D, num_layers=L, num_heads=H, ffn_dim=F,
                                attn_bias=True, activation=Activation.geluTanh, init_std=INIT_STD, **kw))
    elif fam == "llama":
        m = Llama(LlamaConfig(vocab_size=V, max_ctx=c["seq"] + 128, embed_dim=D, num_layers=L, num_heads=H,
                              num_kv_heads=c["kv_heads"], ffn_dim=F, rope_base=ROPE_BASE, init_std=INIT_STD, **kw))
    elif fam == "vit":
        m = ViTClassifier(image_size=c["image"], patch_size=c["patch"], embed_dim=D, num_layers=L, num_heads=H, ffn_dim=F,
                          num_classes=V, activation=Activation.geluTanh, attn_bias=True, init_std=INIT_STD, **kw)
    else:
        m = BertModel(BertConfig(vocab_size=V, max_position_embeddings=c["seq"], embed_dim=D, num_layers=L, num_heads=H,
                                 intermediate_size=F, **kw))
    with torch.no_grad():
        named = {n: weights[n] for n, _, _ in _parameters(c)}
        for p, (n, t) in zip(m.parameters(), named.items(), strict=True):
            p.data.copy_(t.reshape(p.shape))
    return m


# ------------------------------------------------------------------------------------------------ a pass
def prepare(case, seed):
    c = case
    model = _model(c, _weights(c, seed))
    x, y = _inputs(c, seed)
    if c["kind"] == "train":
        opt = dp.Adam(model.parameters(), lr=LR, beta1=BETA1, beta2=BETA2, eps=EPS, weight_decay=DECAY)
        trainer = Trainer(model, opt, clip_norm=CLIP)
        start = opt.arena.flat.clone()
        m, v = _moments(opt.arena.numel, seed)
        for _ in range(3):                     # warm-up, and the step's recording
            trainer.step(x, y)
        # the state a checkpoint of step 1000 would have restored
        opt.arena.flat.copy_(start)
        if opt.arena.master is not None:
            opt.arena.master.copy_(start)
        opt.m.copy_(m)
        opt.v.copy_(v)
        opt._step = RESUMED
        return {"case": c, "trainer": trainer, "opt": opt, "x": x, "y": y}
    model.eval()
    state = {"case": c, "model": model, "x": x}
    if c["kind"] == "decode":
        state["cache"] = _cache(c, model)
        with torch.no_grad():
            model.hidden(x, 0, state["cache"])
        state["next"] = y[:, -1:].contiguous()
    return state


def _cache(c, model):
    return model.new_cache() if c["family"] == "llama" else \
        EncoderCache.empty(c["layers"], c["heads"], max_len=model.config.max_ctx)


def run(state):
    c = state["case"]
    if c["kind"] == "train":
        opt = state["opt"]
        loss = state["trainer"].step(state["x"], state["y"])
        a = opt.arena
        return {"loss": loss, "grad": a.grad, "m": opt.m, "v": opt.v, "weights": a.flat if a.master is None else a.master}
    model = state["model"]
    with torch.no_grad():
        if c["kind"] == "encode":
            return model(state["x"])
        if c["kind"] == "prompt":
            cache = _cache(c, model)
            h = model.hidden(state["x"], 0, cache)
            return {"hidden": h, "logits": ops.linear(h[:, -1], model.head_weight),
                    "k": [layer.k_buf for layer in cache.layers], "v": [layer.v_buf for layer in cache.layers]}
        cache = state["cache"]
        for layer in cache.layers:             # the same step again
            layer.seq_len = c["seq"]
        h = model.hidden(state["next"], c["seq"], cache)
        return {"logits": ops.linear(h[:, -1], model.head_weight),
                "k": [layer.k_buf for layer in cache.layers], "v": [layer.v_buf for layer in cache.layers]}


# ------------------------------------------------------------------------------------------------ what it cannot do without
def work(case):
    c = case
    params = sum(math.prod(s) for _, s, _ in _parameters(c))
    table = sum(math.prod(s) for n, s, _ in _parameters(c) if n in ("tok", "pos"))
    B, S, D, L, V = c["batch"], c["seq"], c["dim"], c["layers"], c["vocab"]
    size = 2 if c["dtype"] == "bf16" else 4
    tied = D * V if c["family"] in ("gpt", "llama") else 0
    tokens = B * S
    causal = c["family"] in ("gpt", "llama")
    attention = 4 * B * S * S * D * L // (2 if causal else 1)
    body = 2 * (params - table)
    kv = 2 * L * c["kv_heads"] * (D // c["heads"]) * size
    if c["kind"] == "train":
        head = 2 * tied * tokens
        flops = 3 * (body * tokens + attention + head)
        # weights read, gradients written; moments and fp32 weights read and written
        return {"bytes": params * (size + size + 24 + (size if size == 2 else 0)), "flops": flops}
    if c["kind"] == "decode":
        return {"bytes": (params - table + tied) * size + kv * B * (S + 1) + B * V * size,
                "flops": B * (body + 2 * tied) + 4 * B * (S + 1) * D * L}
    if c["kind"] == "prompt":
        return {"bytes": (params - table + tied) * size + kv * tokens + tokens * D * size + B * V * size,
                "flops": body * tokens + attention + 2 * tied * B}
    return {"bytes": (params - table) * size + 2 * tokens * D * size, "flops": body * tokens + attention}


def tolerance(case):
    # about four times the distance from ``exact``: 32-bit sums 1.6e-6, bf16 activations and gradients 0.9 to 1.5e-2
    return {"rel": 1e-5} if case["dtype"] == "fp32" else {"rel": 5e-2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rope(x, start):
    """``x [B, heads, S, hd]``, halves rotated against one another."""
    S, hd = x.shape[-2:]
    half = hd // 2
    inv = ROPE_BASE ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    ang = torch.arange(start, start + S, device=x.device, dtype=torch.float64)[:, None] * inv
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def _exact_block(c, w, i, h, past):
    D, H, Hkv = c["dim"], c["heads"], c["kv_heads"]
    hd, fam = D // H, c["family"]
    p = f"{i}."
    B, S = h.shape[:2]

    def norm(x, name):
        if fam == "llama":
            return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w[name + ".g"]
        return TF.layer_norm(x, (D,), w[name + ".g"], w[name + ".b"], 1e-12 if fam == "bert" else 1e-5)

    def linear(x, name):
        return TF.linear(x, w[p + name + ".w"], w.get(p + name + ".b"))

    def heads(x, n):
        return x.reshape(B, S, n, hd).transpose(1, 2)
    x = h if fam == "bert" else norm(h, p + "n1")
    q, k, v = linear(x, "qkv").split([H * hd, Hkv * hd, Hkv * hd], -1)
    q, k, v = heads(q, H), heads(k, Hkv), heads(v, Hkv)
    start = 0 if past is None else past[0].shape[2]
    if fam == "llama":
        q, k = _rope(q, start), _rope(k, start)
    if past is not None:
        k, v = torch.cat([past[0], k], 2), torch.cat([past[1], v], 2)
    kept = (k, v)
    k, v = (t.repeat_interleave(H // Hkv, 1) for t in kept)
    s = q @ k.transpose(-1, -2) / math.sqrt(hd)
    if fam in ("gpt", "llama") and S > 1:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    o = (s.softmax(-1) @ v).transpose(1, 2).reshape(B, S, H * hd)
    h = h + linear(o, "wo")
    if fam == "bert":
        h = norm(h, p + "n1")
    x = h if fam == "bert" else norm(h, p + "n2")
    if fam == "llama":
        g, u = linear(x, "gu").chunk(2, -1)
        h = h + linear(TF.silu(g) * u, "f2")
    else:
        h = h + linear(TF.gelu(linear(x, "f1"), approximate="tanh"), "f2")
    return (norm(h, p + "n2") if fam == "bert" else h), kept


def _exact_stack(c, w, x, pasts=None):
    """Final hidden states and the layers' keys and values; ``pasts``: those of earlier tokens."""
    fam, D = c["family"], c["dim"]
    if fam == "vit":
        B, P, G = c["batch"], c["patch"], c["image"] // c["patch"]
        rows = x.double().reshape(B, 3, G, P, G, P).permute(0, 2, 4, 3, 5, 1).reshape(B, G * G, P * P * 3)
        h = TF.linear(rows, w["patch.w"], w["patch.b"])
        h = torch.cat([w["cls"].expand(B, 1, D), h], 1) + w["pos"]
    else:
        h = w["tok"][x]
        start = 0 if pasts is None else pasts[0][0].shape[2]
        if fam != "llama":
            h = h + w["pos"][start:start + x.shape[1]]
        if fam == "bert":
            h = TF.layer_norm(h + w["type"], (D,), w["ln0.g"], w["ln0.b"], 1e-12)
    kept = []
    for i in range(c["layers"]):
        past = None if pasts is None else pasts[i]
        if torch.is_grad_enabled():
            h = checkpoint(lambda t, i=i: _exact_block(c, w, i, t, None)[0], h, use_reentrant=False)
        else:
            h, kv = _exact_block(c, w, i, h, past)
            kept.append(kv)
    if fam == "llama":
        h = h * torch.rsqrt((h * h).mean(-1, keepdim=True) + 1e-5) * w["lnf.g"]
    elif fam != "bert":
        h = TF.layer_norm(h, (D,), w["lnf.g"], w["lnf.b"], 1e-5)
    return h, kept


def _exact_cache(c, kept):
    """The layers' cache buffers: rows of all heads, room for the whole context in steps of 128 rows, zeros behind."""
    rows = (c["seq"] + 128 + 127) // 128 * 128

    def buffer(t):
        B, Hkv, S, hd = t.shape
        return TF.pad(t.transpose(1, 2).reshape(B, S, Hkv * hd), (0, 0, 0, rows - S))
    return {"k": [buffer(k) for k, _ in kept], "v": [buffer(v) for _, v in kept]}


def exact(case, seed):
    c = case
    w = {n: t.double() for n, t in _weights(c, seed).items()}
    x, y = _inputs(c, seed)
    if c["kind"] != "train":
        with torch.no_grad():
            h, kept = _exact_stack(c, w, x)
            if c["kind"] == "encode":
                return h
            if c["kind"] == "prompt":
                return {"hidden": h, "logits": h[:, -1] @ w["tok"].T, **_exact_cache(c, kept)}
            h, kept = _exact_stack(c, w, y[:, -1:], kept)
            return {"logits": h[:, -1] @ w["tok"].T, **_exact_cache(c, kept)}
    for t in w.values():
        t.requires_grad_(True)
    h, _ = _exact_stack(c, w, x)
    if c["family"] == "vit":
        loss = TF.cross_entropy(TF.linear(h[:, 0], w["head.w"], w["head.b"]), y)
    else:
        loss = TF.cross_entropy(h.reshape(-1, c["dim"]) @ w["tok"].T, y.reshape(-1))
    loss.backward()
    del h
    grad = _arena(c, {n: t.grad for n, t in w.items()}, torch.float64)
    weights = _arena(c, {n: t.detach() for n, t in w.items()}, torch.float64)
    norm = grad.norm()
    g = grad * (CLIP / norm if norm > CLIP else 1.0)
    m, v = (t.double() for t in _moments(grad.numel(), seed))
    m = BETA1 * m + (1 - BETA1) * g
    v = BETA2 * v + (1 - BETA2) * g * g
    t = RESUMED + 1
    step = m / (1 - BETA1 ** t) / ((v / (1 - BETA2 ** t)).sqrt() + EPS)
    return {"loss": loss.detach(), "grad": grad, "m": m, "v": v, "weights": weights - LR * (step + DECAY * weights)}
