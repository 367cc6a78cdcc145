"""Performance cases: what a user of the framework has it do, at the sizes where it is used.

Three kinds of work, each through the entry point that a program calls:

``train``    one optimisation step of ``TrainEngine`` (forward, backward, overflow check, fused AdamW on fp32
             masters, loss-scale update) on a GPT- or Llama-style decoder in bf16.
``prefill``  ``PagedLlamaExecutor.execute_batch`` on requests whose prompts are not cached yet: projections, rotary
             embedding, KV-cache write, causal attention (later chunks of a long prompt attend to their cached
             prefix through the block table), first token.
``decode``   ``PagedLlamaExecutor.execute_batch`` on requests with cached contexts: one token for each.

The decoders have the layer shapes of the package's presets (GPT 1.3 B, Llama 8 B and 13 B) or smaller ones of the same
kind; all but the largest training case have fewer layers than the preset, so that a pass stays short.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from ml_framework_b200.engine import EngineConfig, TrainEngine
from ml_framework_b200.models.gpt import GPT, GPTConfig
from ml_framework_b200.models.llama import Llama, LlamaConfig
from ml_framework_b200.serving.executor import ExecutorConfig, PagedLlamaExecutor
from ml_framework_b200.serving.kv_cache import KVCacheBlockManager
from ml_framework_b200.serving.scheduler import Batch, Request

HEAD = 128                  # head dimension of every preset
PAGE = 16                   # tokens per KV-cache block
VOCAB_PAD = 128
CHUNK = 2048                # prompt tokens of one request that an iteration prefills
POSITIONS = 2048            # learned positions of the GPT models
EPS = 1e-5
THETA = 500000.0
LR, BETAS, ADAM_EPS, DECAY = 3e-4, (0.9, 0.95), 1e-8, 0.1
LOSS_SCALE = 65536.0


# ------------------------------------------------------------------------------------------ the cases
def _train(arch, layers, d, heads, kv_heads, ff, vocab, batch, seq):
    return {"kind": "train", "arch": arch, "layers": layers, "d_model": d, "heads": heads, "kv_heads": kv_heads, "d_ff": ff,
            "vocab": vocab, "batch": batch, "seq": seq}


def _serve(kind, layers, d, heads, kv_heads, ff, vocab, batch, tokens):
    return {"kind": kind, "layers": layers, "d_model": d, "heads": heads, "kv_heads": kv_heads, "d_ff": ff, "vocab": vocab,
            "batch": batch, "tokens": tokens}


_LLAMA_8B = (6, 4096, 32, 8, 14336, 32000)       # layers kept, width, query heads, KV heads, FFN, vocabulary
_LLAMA_13B = (4, 5120, 40, 40, 13824, 32000)


def listed():
    return [
        # The model of the package's smoke run and engine tests: the step is a chain of short launches.
        dict(_train("gpt", 2, 256, 2, 2, 1024, 1000, 2, 256), name="train gpt tiny"),
        # A small GPT on a ragged batch (2331 tokens, no multiple of any tile): fine-tuning on sequences as they come.
        dict(_train("gpt", 4, 1024, 8, 8, 4096, 50257, 3, 777), name="train gpt ragged"),
        # The headline training configuration, whole: GPT 1.3 B, micro-batch 4 x 2048.
        dict(_train("gpt", 24, 2048, 16, 16, 8192, 50257, 4, 2048), name="train gpt 1.3b"),
        # Two layers at Llama 8 B width, sequence 4096: grouped queries, rotary embedding, RMSNorm, SwiGLU, untied head.
        dict(_train("llama", 2, 4096, 32, 8, 14336, 32000, 2, 4096), name="train llama 2 layers"),
        # One short chat turn: latency to the first token.
        dict(_serve("prefill", *_LLAMA_8B, 1, 37), name="prefill 1x37"),
        # Eight requests that arrive together, prompts of 512 tokens: the serving benchmark's shape, prefilled as one batch.
        dict(_serve("prefill", *_LLAMA_8B, 8, 512), name="prefill 8x512"),
        # A long document: three chunks, the later two read their prefix from the paged cache, the last one is ragged.
        dict(_serve("prefill", *_LLAMA_8B, 1, 5500), name="prefill 1x5500"),
        # A single user: latency per token.
        dict(_serve("decode", *_LLAMA_8B, 1, 700), name="decode 1x700"),
        # A moderate, odd batch with longer contexts.
        dict(_serve("decode", *_LLAMA_8B, 13, 2500), name="decode 13x2500"),
        # The serving benchmark's batch.
        dict(_serve("decode", *_LLAMA_8B, 64, 576), name="decode 64x576"),
        # The largest batch that the executor takes by default.
        dict(_serve("decode", *_LLAMA_8B, 256, 1024), name="decode 256x1024"),
        # Multi-head attention without grouping (the 13 B layer shape).
        dict(_serve("decode", *_LLAMA_13B, 24, 900), name="decode mha 24x900"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("train", "prefill", "decode", "decode"))
    if kind == "train":
        arch = rng.choice(("gpt", "llama"))
        d = 256 * _log(rng, 1, 16)
        heads = d // HEAD
        kv = heads
        if arch == "llama" and heads % 4 == 0 and rng.random() < 0.7:
            kv = heads // 4
        ff = 256 * max(2, int(d * rng.uniform(2.5, 4.0)) // 256)
        seq = _log(rng, 64, 2048 if arch == "gpt" else 4096)
        batch = max(1, min(16, _log(rng, 64, 8192) // seq))
        return _train(arch, rng.randint(1, 4), d, heads, kv, ff, rng.choice((1000, 32000, 50257)), batch, seq)
    shape = rng.choice((_LLAMA_8B, _LLAMA_8B, _LLAMA_13B, (6, 2048, 16, 4, 8192, 32000)))
    if kind == "prefill":
        total = _log(rng, 16, 8192)
        batch = rng.choice((1, 1, 2, 4, 7))
        return _serve("prefill", *shape, batch, max(8, total // batch))
    batch = _log(rng, 1, 256)
    return _serve("decode", *shape, batch, _log(rng, 32, max(64, min(4000, 262144 // batch * 4096 // (shape[3] * 1024) // 2))))


# ------------------------------------------------------------------------------------------ inputs from the seed
def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def _padded(vocab):
    return (vocab + VOCAB_PAD - 1) // VOCAB_PAD * VOCAB_PAD


def _shapes(c):
    """(name, shape, standard deviation or None for ones) of every weight, in the models' parameter order."""
    d, f, L, V = c["d_model"], c["d_ff"], c["layers"], _padded(c["vocab"])
    std = 0.02
    out_std = std / (2 * L) ** 0.5
    q = c["heads"] * HEAD
    if c["kind"] == "train" and c["arch"] == "gpt":
        s = [("embed.weight", (V, d), std), ("embed.pos_weight", (POSITIONS, d), std)]
        for i in range(L):
            p = f"blocks.{i}."
            s += [(p + "ln1.weight", (d,), None), (p + "ln1.bias", (d,), std), (p + "attn.qkv.weight", (3 * q, d), std),
                  (p + "attn.qkv.bias", (3 * q,), std), (p + "attn.proj.weight", (d, q), out_std), (p + "attn.proj.bias", (d,), std),
                  (p + "ln2.weight", (d,), None), (p + "ln2.bias", (d,), std), (p + "mlp.fc1.weight", (f, d), std),
                  (p + "mlp.fc1.bias", (f,), std), (p + "mlp.fc2.weight", (d, f), out_std), (p + "mlp.fc2.bias", (d,), std)]
        return s + [("ln_f.weight", (d,), None), ("ln_f.bias", (d,), std)]
    kv = c["kv_heads"] * HEAD
    # A served model is a trained one, whose next token is mostly a clear winner: its embedding dominates the residual
    # stream and the head points from each token to another one. A fresh one (train) has small random weights.
    s = [("lm_head", (V, d), std), ("embed.weight", (V, d), 1.0 if c["kind"] != "train" else std)]
    for i in range(L):
        p = f"blocks.{i}."
        s += [(p + "norm1.weight", (d,), None), (p + "attn.qkv.weight", (q + 2 * kv, d), std), (p + "attn.proj.weight", (d, q), out_std),
              (p + "norm2.weight", (d,), None), (p + "mlp.gate_up.weight", (2 * f, d), std), (p + "mlp.down.weight", (d, f), out_std)]
    return s + [("norm_f.weight", (d,), None)]


def _weights(c, seed):
    g = _gen(seed)
    w = {}
    for name, shape, std in _shapes(c):
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        w[name] = t.normal_(1.0, 0.05, generator=g) if std is None else t.normal_(0.0, std, generator=g)
    if c["kind"] != "train":
        w["lm_head"].copy_(w["embed.weight"].roll(1, 0) * 0.02)
    return w


def _lengths(c):
    """Cached tokens of each request before a decode step: from half of ``tokens`` up to it."""
    n = c["tokens"]
    return [n - (i * 37) % (n // 2 + 1) for i in range(c["batch"])]


def _pages(n):
    return (n + PAGE - 1) // PAGE


def _prompts(c, seed):
    return torch.randint(1, c["vocab"], (c["batch"], c["tokens"]), generator=_gen(seed, 1), device="cuda")


def _last_tokens(c, seed):
    return torch.randint(1, c["vocab"], (c["batch"],), generator=_gen(seed, 1), device="cuda")


def _batch_ids(c, seed):
    return torch.randint(0, c["vocab"], (2, c["batch"], c["seq"]), generator=_gen(seed, 1), device="cuda")


def _fill_cache(cache, seed, layer):
    """Cached keys and values of earlier tokens: unit normal, as projections of normalised activations are."""
    cache.normal_(0.0, 1.0, generator=_gen(seed, 100 + layer))


def _cache_pages(c):
    if c["kind"] == "prefill":
        return c["batch"] * _pages(c["tokens"])
    return sum(_pages(n + 1) for n in _lengths(c))


def prepare(case, seed):
    c = case
    w = _weights(c, seed)
    if c["kind"] == "train":
        if c["arch"] == "gpt":
            model = GPT(GPTConfig(c["layers"], c["d_model"], c["heads"], c["d_ff"], c["vocab"], POSITIONS), torch.bfloat16, "cuda")
        else:
            model = Llama(LlamaConfig(c["layers"], c["d_model"], c["heads"], c["kv_heads"], HEAD, c["d_ff"], c["vocab"], c["seq"], THETA),
                          torch.bfloat16, "cuda")
        _load(model, w)
        eng = TrainEngine(model, EngineConfig(lr=LR, betas=BETAS, eps=ADAM_EPS, weight_decay=DECAY))
        ids, targets = _batch_ids(c, seed)
        return {"case": c, "engine": eng, "ids": ids, "targets": targets}
    model = Llama(LlamaConfig(c["layers"], c["d_model"], c["heads"], c["kv_heads"], HEAD, c["d_ff"], c["vocab"], 8192, THETA),
                  torch.bfloat16, "cuda").eval()
    _load(model, w)
    kv = KVCacheBlockManager(_cache_pages(c), PAGE, HEAD, c["layers"], c["kv_heads"], device="cuda", dtype=torch.bfloat16)
    ex = PagedLlamaExecutor(model, kv, ExecutorConfig(max_seq_len=8192 if c["kind"] == "prefill" else 4096, prefill_chunk=CHUNK))
    if c["kind"] == "prefill":
        reqs = [Request(p, max_tokens=1, id=i) for i, p in enumerate(_prompts(c, seed).tolist())]
        return {"case": c, "executor": ex, "kv": kv, "requests": reqs}
    lens = _lengths(c)
    for i, n in enumerate(lens):
        kv.append_tokens(i, n)
    for layer, cache in enumerate(kv.caches):
        _fill_cache(cache, seed, layer)
    reqs = [Request([1] * n, max_tokens=64, id=i, generated=[t], prefilled=n) for i, (n, t) in enumerate(zip(lens, _last_tokens(c, seed).tolist()))]
    return {"case": c, "executor": ex, "kv": kv, "requests": reqs, "lengths": lens}


@torch.no_grad()
def _load(model, w):
    named = dict(model.named_parameters())
    assert named.keys() == w.keys(), sorted(named.keys() ^ w.keys())
    for name, t in w.items():
        named[name].copy_(t)


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["case"]["kind"]
    if kind == "train":
        eng = state["engine"]
        loss = eng.step(state["ids"], state["targets"])
        opt = eng.optimizer.segments[0]
        return {"loss": loss.detach(), "grad": eng.flat.grad, "weights": eng.flat.flat, "master": opt.master, "m": opt.m, "v": opt.v}
    ex, kv, reqs = state["executor"], state["kv"], state["requests"]
    if kind == "prefill":
        # every chunk of every prompt, as the scheduler hands the executor unfinished prompts iteration by iteration
        tokens = {}
        for r in reqs:
            r.prefilled = 0
        while len(tokens) < len(reqs):
            tokens.update(ex.execute_batch(Batch(reqs, prefill=[r for r in reqs if r.id not in tokens])).generated_tokens)
        for r in reqs:                       # each request asked for one token: its pages go back to the pool
            kv.free_sequence_blocks(r.id)
    else:
        tokens = ex.execute_batch(Batch(reqs, decode=reqs)).generated_tokens
        for r, n in zip(reqs, state["lengths"]):
            kv.truncate(r.id, n)             # the token is not kept, so that every pass is the same step
    return {"tokens": np.array([tokens[r.id] for r in reqs]), "cache": list(kv.caches)}


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _matmul_params(c):
    d, q = c["d_model"], c["heads"] * HEAD
    mlp = 2 * d * c["d_ff"] if c.get("arch") == "gpt" else 3 * d * c["d_ff"]
    return c["layers"] * (d * (q + 2 * c["kv_heads"] * HEAD) + q * d + mlp)


def work(case):
    c = case
    d, V, L, q = c["d_model"], _padded(c["vocab"]), c["layers"], c["heads"] * HEAD
    P = _matmul_params(c)
    if c["kind"] == "train":
        T = c["batch"] * c["seq"]
        params = sum(math.prod(s) for _, s, _ in _shapes(c))
        attn = 2 * 2 * T * (c["seq"] / 2) * q * L
        # masters and both moments read and written, bf16 weights read and written, gradients written
        return {"bytes": params * (24.0 + 4 + 2) + 16.0 * T, "flops": 3 * (2.0 * T * (P + d * V) + attn)}
    kv_row = 2 * c["kv_heads"] * HEAD * 2 * L               # cache bytes of one token over all layers
    weights = 2.0 * (P + d * V)
    if c["kind"] == "prefill":
        T = c["batch"] * c["tokens"]
        return {"bytes": weights + T * (kv_row + 2 * d), "flops": 2.0 * T * P + 2 * 2 * T * (c["tokens"] / 2) * q * L + 2.0 * c["batch"] * d * V}
    ctx = sum(n + 1 for n in _lengths(c))
    return {"bytes": weights + ctx * kv_row + c["batch"] * 2 * d, "flops": 2.0 * c["batch"] * (P + d * V) + 4.0 * ctx * q * L}


def tolerance(case):
    # bf16 activations, rounded between operators and, where few rows are split over the SMs, between partial sums.
    # Against `exact`: gradients and their moments up to 0.020, cached keys and values up to 0.022 in the last layer; the
    # single largest difference of one value stays below 0.62 (train) and 0.16 (serve) of the root mean square.
    return {"rel": 0.03, "max": 0.99} if case["kind"] == "train" else {"rel": 0.03, "max": 0.6, "differ": 0.0}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, g):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * g


def _rope(x, pos):
    """x [T, heads, 128]: pairs (i, i + 64) turned by pos / theta^(2 i / 128)."""
    half = HEAD // 2
    f = THETA ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / HEAD)
    a = pos.double()[:, None, None] * f
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _attend(q, k, v):
    """Causal attention of one sequence: q [S, Hq, 128], k, v [S, Hkv, 128]; a few heads at a time."""
    S, Hq, _ = q.shape
    rep = Hq // k.shape[1]
    mask = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1)
    out = []
    step = max(1, (1 << 28) // (S * S))
    for h in range(0, Hq, step):
        hs = torch.arange(h, min(h + step, Hq), device=q.device)
        s = torch.einsum("qhd,khd->hqk", q[:, hs], k[:, hs // rep]) * HEAD ** -0.5
        out.append(torch.einsum("hqk,khd->qhd", s.masked_fill(mask, float("-inf")).softmax(-1), v[:, hs // rep]))
    return torch.cat(out, 1)


def _swiglu(h, gate_up):
    t = h @ gate_up.T
    return F.silu(t[:, 0::2]) * t[:, 1::2]


def _train_block(c, x, w, pre):
    B, S = c["batch"], c["seq"]
    q, kv = c["heads"] * HEAD, c["kv_heads"] * HEAD
    gpt = c["arch"] == "gpt"
    d = x.shape[-1]
    if gpt:
        h = F.layer_norm(x, (d,), w[pre + "ln1.weight"], w[pre + "ln1.bias"], EPS)
        t = F.linear(h, w[pre + "attn.qkv.weight"], w[pre + "attn.qkv.bias"])
    else:
        t = F.linear(_rms(x, w[pre + "norm1.weight"]), w[pre + "attn.qkv.weight"])
    Q, K, V = (u.reshape(B * S, -1, HEAD) for u in t.split([q, kv, kv], -1))
    if not gpt:
        pos = torch.arange(S, device=x.device).repeat(B)
        Q, K = _rope(Q, pos), _rope(K, pos)
    a = torch.cat([checkpoint(_attend, Q[i:i + S], K[i:i + S], V[i:i + S], use_reentrant=False) for i in range(0, B * S, S)])
    if gpt:
        x = x + F.linear(a.reshape(B * S, q), w[pre + "attn.proj.weight"], w[pre + "attn.proj.bias"])
        h = F.layer_norm(x, (d,), w[pre + "ln2.weight"], w[pre + "ln2.bias"], EPS)
        h = F.gelu(F.linear(h, w[pre + "mlp.fc1.weight"], w[pre + "mlp.fc1.bias"]), approximate="tanh")
        return x + F.linear(h, w[pre + "mlp.fc2.weight"], w[pre + "mlp.fc2.bias"])
    x = x + F.linear(a.reshape(B * S, q), w[pre + "attn.proj.weight"])
    return x + F.linear(_swiglu(_rms(x, w[pre + "norm2.weight"]), w[pre + "mlp.gate_up.weight"]), w[pre + "mlp.down.weight"])


def _flat(tensors):
    """One buffer, each tensor at a multiple of 8 elements: the layout of the engine's parameter and gradient buffers."""
    n = sum((t.numel() + 7) // 8 * 8 for t in tensors)
    out, at = torch.zeros(n, dtype=torch.float64, device="cuda"), 0
    for t in tensors:
        out[at:at + t.numel()] = t.detach().reshape(-1)
        at += (t.numel() + 7) // 8 * 8
    return out


def _exact_train(c, seed):
    w = {k: t.double().requires_grad_() for k, t in _weights(c, seed).items()}
    ids, targets = _batch_ids(c, seed)
    x = w["embed.weight"][ids.reshape(-1)]
    if c["arch"] == "gpt":
        x = x + w["embed.pos_weight"][:c["seq"]].repeat(c["batch"], 1)
    for i in range(c["layers"]):
        x = checkpoint(_train_block, c, x, w, f"blocks.{i}.", use_reentrant=False)
    if c["arch"] == "gpt":
        h, head = F.layer_norm(x, (c["d_model"],), w["ln_f.weight"], w["ln_f.bias"], EPS), w["embed.weight"]
    else:
        h, head = _rms(x, w["norm_f.weight"]), w["lm_head"]
    loss = F.cross_entropy(h @ head[:c["vocab"]].T, targets.reshape(-1))
    loss.backward()
    grad = _flat([t.grad for t in w.values()])
    for t in w.values():
        t.grad = None
    p = _flat(list(w.values()))
    w.clear()
    m, v = (1 - BETAS[0]) * grad, (1 - BETAS[1]) * grad * grad
    p -= LR * DECAY * p
    p -= LR * grad / (grad.abs() + ADAM_EPS)       # first step: m and v without their bias are the gradient and its square
    grad *= LOSS_SCALE
    return {"loss": loss.detach(), "grad": grad, "weights": p, "master": p, "m": m, "v": v}


@torch.no_grad()
def _exact_serve(c, seed):
    w = {k: t.double() for k, t in _weights(c, seed).items()}
    B, q, kv = c["batch"], c["heads"] * HEAD, c["kv_heads"]
    prefill = c["kind"] == "prefill"
    lens = [0] * B if prefill else _lengths(c)
    new = c["tokens"] if prefill else 1
    ids = (_prompts(c, seed) if prefill else _last_tokens(c, seed)[:, None]).reshape(-1)
    pos = torch.cat([torch.arange(n, n + new, device="cuda") for n in lens])
    pages = _cache_pages(c)
    # pages are handed out in order: each request's cached tokens first, then what the new tokens need, chunk by chunk
    table, used = [[] for _ in lens], 0
    for begin in [-CHUNK] + list(range(0, new, CHUNK)):
        for t, n in zip(table, lens):
            more = _pages(n + max(0, min(begin + CHUNK, new))) - len(t)
            t += range(used, used + more)
            used += more
    tables = [torch.tensor(t, device="cuda") for t in table]
    caches = []
    x = w["embed.weight"][ids]
    for i in range(c["layers"]):
        pre = f"blocks.{i}."
        cache = torch.zeros(pages, 2, PAGE, kv, HEAD, dtype=torch.bfloat16, device="cuda")
        if not prefill:
            _fill_cache(cache, seed, i)
        cache = cache.double()
        t = _rms(x, w[pre + "norm1.weight"]) @ w[pre + "attn.qkv.weight"].T
        Q, K, V = (u.reshape(-1, u.shape[-1] // HEAD, HEAD) for u in t.split([q, kv * HEAD, kv * HEAD], -1))
        Q, K = _rope(Q, pos), _rope(K, pos)
        a = []
        for r in range(B):
            rows = slice(r * new, (r + 1) * new)
            at = pos[rows]
            cache[tables[r][at // PAGE], 0, at % PAGE] = K[rows]
            cache[tables[r][at // PAGE], 1, at % PAGE] = V[rows]
            if prefill:
                a.append(_attend(Q[rows], K[rows], V[rows]))
                continue
            n = lens[r] + 1
            k, v = (cache[tables[r], j].reshape(-1, kv, HEAD)[:n] for j in (0, 1))
            qq = Q[r].reshape(kv, -1, HEAD)
            s = torch.einsum("hgd,nhd->hgn", qq, k) * HEAD ** -0.5
            a.append(torch.einsum("hgn,nhd->hgd", s.softmax(-1), v).reshape(1, -1, HEAD))
        caches.append(cache)
        x = x + torch.cat(a).reshape(B * new, q) @ w[pre + "attn.proj.weight"].T
        x = x + _swiglu(_rms(x, w[pre + "norm2.weight"]), w[pre + "mlp.gate_up.weight"]) @ w[pre + "mlp.down.weight"].T
    last = _rms(x[new - 1::new], w["norm_f.weight"])
    tokens = (last @ w["lm_head"][:c["vocab"]].T).argmax(-1).cpu().numpy()
    return {"tokens": tokens, "cache": caches}


def exact(case, seed):
    return _exact_train(case, seed) if case["kind"] == "train" else _exact_serve(case, seed)
