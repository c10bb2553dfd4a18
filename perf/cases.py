"""What the framework's speed is measured on: steps of a serving engine and calls of the embedding
engine, at the sizes of the serving, layer and embedding benchmarks.

Four paths:

    embed     ``EmbeddingEngine.encode`` of the BERT-base architecture: token lists on the host in,
              pooled vectors on the host out
    llama     one engine step of the Llama-3.1-8B architecture (or its SwiftKV variant) through
              ``ModelRunner.score``: prompt chunks, decodes, drafts to verify, or a mix of them, over
              the paged cache; out come the logits of the sampled rows and the cache
    taralix   the same for latent attention and routed experts (the layer benchmark's moe-2048)
    fp8       the feed-forward halves of fp8 layers at the Llama-3.1-8B widths as the serving
              benchmark runs them: norm and quantisation, gate / up, activation and quantisation,
              down; steps of up to 512 tokens are captured, as the engine captures them. (Whole fp8
              models have no case of their own: a change of one rounding in attention, which is no
              error, moves the logits of a random fp8 model by several per cent.)

The models have their full widths but few layers and a vocabulary of 32000, so that a state is made in
about a second; every layer does the same work, so what a step costs per layer is what it costs in
the whole model. Weights, cached keys and values and tokens are random and made from the seed; weights
have the variance of a random checkpoint.

Lengths are ragged: ``lengths`` spreads them by a quarter around their mean, the same way for equal
numbers, so that the work of a case follows from its numbers alone.
"""

from __future__ import annotations

import dataclasses
import math
import os

import numpy as np
import torch

os.environ.setdefault("AB200_GC_FREEZE", "0")    # engines come and go in this process

VOCAB, BLOCK = 32000, 64
HIDDEN, HEADS, KV_HEADS, DIM, FF = 4096, 32, 8, 128, 14336      # Llama-3.1-8B
T_WIDTH, T_HEADS, T_DIM, T_RANK = 2048, 16, 128, 512             # layer benchmark, moe-2048
T_FF, T_EXPERTS, T_TOP, T_ALPHA = 1408, 64, 6, 1.5
B_WIDTH, B_HEADS, B_FF, B_LAYERS, B_VOCAB = 768, 12, 3072, 12, 30522   # BERT-base


def _embed(texts, tokens, ragged=True):
    return {"path": "embed", "texts": texts, "tokens": tokens, "ragged": ragged}


def _step(path, layers, swiftkv=False, decodes=0, context=0, drafts=0, prompts=0, prompt=0, cached=0):
    return {"path": path, "layers": layers, "swiftkv": swiftkv, "decodes": decodes,
            "context": context, "drafts": drafts, "prompts": prompts, "prompt": prompt,
            "cached": cached}


def _fp8(tokens):
    return {"path": "fp8", "layers": 2, "tokens": tokens}


def listed():
    return [
        # a search query is embedded on its own: latency and launches
        {"name": "embed_one", **_embed(1, 50, False)},
        # short texts in bulk (the embedding benchmark's length 50)
        {"name": "embed_short", **_embed(1024, 50)},
        # documents at the encoder's full length (the embedding benchmark's length 512)
        {"name": "embed_long", **_embed(64, 512, False)},
        # one user: a chat continues token by token
        {"name": "decode_one", **_step("llama", 4, decodes=1, context=700)},
        # the serving benchmark's decode step: 128 requests of 2000 tokens
        {"name": "decode_batch", **_step("llama", 4, decodes=128, context=2000)},
        # speculation: every request verifies three drafted tokens
        {"name": "verify_drafts", **_step("llama", 4, decodes=24, context=3000, drafts=3)},
        # the serving benchmark's prefill step: a token budget of 8192 in prompts of about 2000
        {"name": "prefill_batch", **_step("llama", 2, prompts=4, prompt=2048)},
        # a chunk of a long document: 8192 tokens behind 24576 that are cached
        {"name": "prefill_long", **_step("llama", 2, prompts=1, prompt=8192, cached=24576)},
        # chunked prefill beside decodes, SwiftKV
        {"name": "mixed_swiftkv", **_step("llama", 4, swiftkv=True, decodes=61, context=1500, prompts=1,
                                          prompt=1987)},
        # fp8 serving: the linears of a prefill step and of a decode step
        {"name": "fp8_prefill", **_fp8(8192)},
        {"name": "fp8_decode", **_fp8(128)},
        # latent attention and routed experts
        {"name": "experts_prefill", **_step("taralix", 2, prompts=4, prompt=2048)},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["embed", "embed", "embed", "decode", "decode", "decode", "prefill", "prefill",
                       "long", "mixed", "fp8", "fp8", "experts_prefill", "experts_decode"])
    if kind == "embed":
        tokens = _log(rng, 8, 512)
        return _embed(_log(rng, 1, max(1, 52000 // tokens)), tokens, rng.random() < 0.7)
    if kind == "fp8":
        return _fp8(_log(rng, 1, 8192))
    if kind == "decode":
        drafts = rng.choice([0, 0, 0, 1, 3])
        n = _log(rng, 1, 200 // (drafts + 1))
        return _step("llama", 4, decodes=n, drafts=drafts, context=_log(rng, 64, min(16000, 256000 // n)))
    if kind == "prefill":
        n = rng.randint(1, 12)
        return _step("llama", 2, prompts=n, prompt=_log(rng, 40, 8192 // n))
    if kind == "long":
        return _step("llama", 2, prompts=1, prompt=_log(rng, 512, 8192), cached=_log(rng, 1000, 24576))
    if kind == "mixed":
        swiftkv = rng.random() < 0.5
        return _step("llama", 4 if swiftkv else 2, swiftkv=swiftkv, decodes=rng.randint(1, 100),
                     context=_log(rng, 100, 2500), prompts=rng.randint(1, 3), prompt=_log(rng, 100, 2500))
    if kind == "experts_prefill":
        n = rng.randint(1, 8)
        return _step("taralix", 2, prompts=n, prompt=_log(rng, 64, 8192 // n))
    n = _log(rng, 1, 160)
    return _step("taralix", 2, decodes=n, context=_log(rng, 64, 3000))


# ------------------------------------------------------------------------------ sizes
def lengths(n, mean, spread=0.25, most=None):
    """n lengths around ``mean``, the same for the same numbers."""
    out = [max(1, int(mean * (1 + spread * (2 * ((0.5 + 0.6180339887 * i) % 1.0) - 1)))) for i in range(n)]
    return out if most is None else [min(x, most) for x in out]


def text_lengths(c):
    return lengths(c["texts"], c["tokens"], 0.25 if c["ragged"] else 0.0, 512)


def spans(c):
    """(cached tokens, new tokens, sampled rows) of every request of a step."""
    out = [(n - 1 - c["drafts"] if n > c["drafts"] else 0, 1 + c["drafts"], 1 + c["drafts"])
           for n in lengths(c["decodes"], c["context"])]
    return out + [(c["cached"], n, 1) for n in lengths(c["prompts"], c["prompt"])]


def blocks_of(c):
    """The first cache block of every request, and the number of blocks."""
    first, at = [], 1
    for cached, new, _ in spans(c):
        first.append(at)
        at += -(-(cached + new) // BLOCK)
    return first, at


def kv_layers(c):
    return c["layers"] // 2 if c["swiftkv"] else c["layers"]


# ---------------------------------------------------------------------------- prepare
def llama_config(c):
    from arcticinference_b200.config import PRESETS
    more = {"num_key_value_layers": kv_layers(c)} if c["swiftkv"] else {}
    return dataclasses.replace(PRESETS["llama-3.1-8b-swiftkv" if c["swiftkv"] else "llama-3.1-8b"],
                               num_hidden_layers=c["layers"], vocab_size=VOCAB, **more)


def taralix_config(c):
    from arcticinference_b200.config import ModelConfig
    layers = []
    for i in range(c["layers"]):
        m = {"heads": T_HEADS, "dim": T_DIM, "vdim": T_DIM, "kv_rank": T_RANK, "scale": T_DIM ** -0.5}
        if i % 2:
            m["kv_from"] = i - 1
        layers.append({"type": "latent_attention", "mixer": m, "mlp": {
            "kind": "moe", "expert": {"ff": T_FF}, "router": {"experts": T_EXPERTS, "top": T_TOP}}})
    return ModelConfig.from_layer_list({"architecture": "Taralix", "width": T_WIDTH, "vocab": VOCAB,
                                        "norm": {"eps": 1e-6}, "postln_alpha": T_ALPHA, "layers": layers})


def tokens_of(c, seed):
    rng = np.random.default_rng(seed)
    if c["path"] == "embed":
        return [rng.integers(0, B_VOCAB, n) for n in text_lengths(c)]
    return [rng.integers(0, VOCAB, cached + new) for cached, new, _ in spans(c)]


def fill_cache(tensors, seed):
    """What earlier steps left in the cache."""
    gen = torch.Generator(device="cuda")
    for i, t in enumerate(tensors):
        gen.manual_seed(1000 * seed + 17 + i)
        t.normal_(generator=gen)


def cache_tensors(runner):
    runs = getattr(runner.kv, "runs", None)
    if runs is not None:      # (layers that share latents share a tensor)
        return list({t.data_ptr(): t for run in runs for t in run}.values())
    return [t for pair in zip(runner.kv.k, runner.kv.v) for t in pair]


def fp8_inputs(c, seed):
    """(activations, residual stream, [(norm, gate | up, down)])"""
    rnd = Weights(seed)
    return rnd(1, c["tokens"], HIDDEN, std=0.5), rnd(2, c["tokens"], HIDDEN, std=1.0), \
        [(1.0 + rnd(10 * l + 3, HIDDEN, std=0.1), rnd(10 * l + 4, 2 * FF, HIDDEN), rnd(10 * l + 5, HIDDEN, FF))
         for l in range(c["layers"])]


def feed_forwards(state):
    from arcticinference_b200 import ops
    h, residual = state["x"], state["residual"].clone()
    for norm, gate_up, down in state["weights"]:
        x = ops.rmsnorm(h, norm, 1e-5, residual=residual, quant=True)
        h = ops.linear(ops.silu_mul_blocked(ops.linear(x, gate_up), quant=True), down)
    return {"out": h, "residual": residual}


def prepare_fp8(case, seed):
    from arcticinference_b200 import ops
    from arcticinference_b200.models.quant import quantize_weight_fp8_row
    x, residual, weights = fp8_inputs(case, seed)
    weights = [(n, quantize_weight_fp8_row(g), quantize_weight_fp8_row(d)) for n, g, d in weights]
    for _, g, d in weights:
        ops.mark_static(g)       # parameters, as in a loaded model
        ops.mark_static(d)
    state = {"path": "fp8", "x": x, "residual": residual, "weights": weights, "graph": None}
    if case["tokens"] <= 512:
        feed_forwards(state)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["result"] = feed_forwards(state)
    return state


def prepare(case, seed):
    seed = seed % 100003
    if case["path"] == "fp8":
        return prepare_fp8(case, seed)
    if case["path"] == "embed":
        from arcticinference_b200.embedding.engine import EmbeddingEngine
        return {"path": "embed", "engine": EmbeddingEngine("bert-base", seed=seed),
                "texts": tokens_of(case, seed)}
    from arcticinference_b200.config import (CacheConfig, EngineConfig, ParallelConfig,
                                             SchedulerConfig)
    from arcticinference_b200.engine.llm_engine import LLMEngine
    from arcticinference_b200.engine.request import Request
    from arcticinference_b200.engine.sampling_params import SamplingParams
    from arcticinference_b200.engine.scheduler import ScheduledRequest, SchedulerOutput
    todo = spans(case)
    first, blocks = blocks_of(case)
    longest = max(cached + new for cached, new, _ in todo)
    config = EngineConfig(
        model=llama_config(case) if case["path"] == "llama" else taralix_config(case),
        parallel=ParallelConfig(),
        cache=CacheConfig(block_size=BLOCK, num_gpu_blocks=blocks, enable_prefix_caching=False),
        scheduler=SchedulerConfig(max_model_len=-(-longest // BLOCK) * BLOCK,
                                  max_num_seqs=max(256, len(todo))),
        load_format="dummy", seed=seed)
    engine = LLMEngine(config, device="cuda")
    fill_cache(cache_tensors(engine.runner), seed)
    step = SchedulerOutput()
    for i, (ids, (cached, new, sampled)) in enumerate(zip(tokens_of(case, seed), todo)):
        r = Request("r%d" % i, ids.tolist(), SamplingParams(temperature=0.0, ignore_eos=True))
        r.block_ids = list(range(first[i], first[i] + -(-(cached + new) // BLOCK)))
        step.scheduled.append(ScheduledRequest(r, cached, new, sampled - 1, True,
                                               want=list(range(new - sampled, new))))
        step.total_tokens += new
    engine.runner.score(step)      # an engine that serves has captured its steps
    return {"path": case["path"], "engine": engine, "step": step}


def run(state):
    if state["path"] == "fp8":
        if state["graph"] is None:
            return feed_forwards(state)
        state["graph"].replay()
        return state["result"]
    engine = state["engine"]
    if state["path"] == "embed":
        return {"vectors": engine.encode(state["texts"])}
    with torch.inference_mode():
        logits = engine.runner.score(state["step"])
    return {"logits": logits, "cache": cache_tensors(engine.runner)}


# ------------------------------------------------------------------------------- work
def work(case):
    if case["path"] == "embed":
        lens = text_lengths(case)
        t = sum(lens)
        layer = 4 * B_WIDTH * B_WIDTH + 2 * B_WIDTH * B_FF
        rows = min(t, B_VOCAB) + min(512, t)
        return {"bytes": 2 * B_LAYERS * layer + 2 * B_WIDTH * rows + 16 * t + 4 * B_WIDTH * len(lens),
                "flops": B_LAYERS * (2 * t * layer + sum(4 * n * n * B_WIDTH for n in lens))}
    if case["path"] == "fp8":
        t, w, n = case["tokens"], 3 * HIDDEN * FF, case["layers"]
        return {"bytes": n * w + 12 * t * HIDDEN, "flops": n * 2 * t * w}
    todo = spans(case)
    t = sum(new for _, new, _ in todo)
    rows = sum(s for _, _, s in todo)
    # (query, key) pairs that attend; keys that a step reads
    pairs = sum(new * cached + new * (new + 1) // 2 for cached, new, _ in todo)
    keys = sum(cached + new for cached, new, _ in todo)
    if case["path"] == "llama":
        q, kv, mlp = HEADS * DIM * HIDDEN, KV_HEADS * DIM * HIDDEN, 3 * HIDDEN * FF
        n = kv_layers(case)
        later = case["layers"] - n
        late_pairs = sum(s * (cached + new) - s * (s - 1) // 2 for cached, new, s in todo)
        flops = n * (2 * t * (2 * q + 2 * kv + mlp) + 4 * pairs * HEADS * DIM) + 2 * rows * VOCAB * HIDDEN
        flops += later * (4 * t * kv + 2 * rows * (2 * q + mlp) + 4 * late_pairs * HEADS * DIM)
        nbytes = case["layers"] * (2 * (2 * q + 2 * kv + mlp) + 4 * keys * KV_HEADS * DIM)
        nbytes += 2 * VOCAB * HIDDEN + 2 * t * HIDDEN + 2 * rows * VOCAB
        return {"bytes": nbytes, "flops": flops}
    used = T_EXPERTS * (1 - (1 - T_TOP / T_EXPERTS) ** t)      # experts that any token chose
    expert, hd = 3 * T_WIDTH * T_FF, T_HEADS * T_DIM
    owned = (case["layers"] + 1) // 2
    maps = 2 * hd * T_WIDTH + 2 * hd * T_RANK + T_EXPERTS * T_WIDTH
    flops = case["layers"] * (2 * t * (maps + T_TOP * expert) + 4 * pairs * hd) + \
        owned * 2 * t * T_RANK * T_WIDTH + 2 * rows * VOCAB * T_WIDTH
    nbytes = 2 * case["layers"] * (maps + used * expert + keys * T_RANK) + 2 * owned * T_RANK * T_WIDTH
    return {"bytes": nbytes + 2 * VOCAB * T_WIDTH + 2 * t * T_WIDTH + 2 * rows * VOCAB, "flops": flops}


def tolerance(case):
    # measured: other orders of the attention's sums move the logits by 0.011 and the encoder's
    # vectors, which are 0.011 from the 64-bit ones, by as much
    return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------ exact
class Weights:
    """The random checkpoint's matrices by the number of their draw."""

    def __init__(self, seed):
        self.seed, self.gen, self.count = seed, torch.Generator(device="cuda"), 0

    def __call__(self, tag, *shape, std=0.02):
        self.gen.manual_seed(self.seed * 1000003 + tag)
        t = torch.randn(shape, generator=self.gen, device="cuda", dtype=torch.float32)
        return (t * std).to(torch.bfloat16)

    def next(self, *shape, std=None):
        self.count += 1
        return self(self.count, *shape, std=shape[-1] ** -0.5 if std is None else std)


def f64(t):
    return t.to(torch.float64)


def e4m3(w):
    """The matrix that fp8 codes with one scale per row stand for."""
    w = w.float()
    scale = w.abs().amax(dim=1, keepdim=True).clamp_min(1e-10) / 448.0
    return f64((w / scale).clamp(-448, 448).to(torch.float8_e4m3fn)) * f64(scale)


def e4m3_rows(x):
    """Activations as a product with fp8 weights takes them: fp8 codes, one scale per token."""
    scale = x.abs().amax(-1, keepdim=True).clamp_min(1e-10) / 448.0
    return f64((x / scale).float().to(torch.float8_e4m3fn)) * scale


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def attend(q, k, v, scale, causal=True):
    """q [n, H, d], k [m, G, d], v [m, G, e]; the queries are the last n positions. [n, H * e]"""
    n, m, G = q.shape[0], k.shape[0], k.shape[1]
    k, v = k.permute(1, 2, 0), v.permute(1, 0, 2)
    out = []
    step = max(1, int(2e8) // (m * q.shape[1]))
    for a in range(0, n, step):
        part = q[a:a + step]
        r = part.shape[0]
        s = part.view(r, G, -1, q.shape[2]).permute(1, 2, 0, 3).reshape(G, -1, q.shape[2]) @ k * scale
        if causal:
            last = torch.arange(m - n + a, m - n + a + r, device="cuda").repeat(s.shape[1] // r)
            s.masked_fill_(torch.arange(m, device="cuda")[None, :] > last[:, None], -math.inf)
        o = (torch.softmax(s, -1) @ v).view(G, -1, r, v.shape[2])
        out.append(o.permute(2, 0, 1, 3).reshape(r, -1))
    return torch.cat(out)


def exact_llama(c, seed):
    eps, rnd = 1e-5, Weights(seed)
    todo, ids = spans(c), tokens_of(c, seed)
    first, blocks = blocks_of(c)
    cache = [torch.empty(blocks, KV_HEADS, BLOCK, DIM, dtype=torch.bfloat16, device="cuda")
             for _ in range(2 * c["layers"])]
    fill_cache(cache, seed)
    cache = [f64(t) for t in cache]
    def lin(x, w):
        return x @ f64(w).t()

    inv = 500000.0 ** -(torch.arange(0, DIM, 2, dtype=torch.float64) / DIM)
    smooth = (8192 * inv / (2 * math.pi) - 1.0) / 3.0
    inv = torch.where(smooth < 0, inv / 8, torch.where(smooth > 1, inv, (1 - smooth) * inv / 8 + smooth * inv))
    new = torch.as_tensor(np.concatenate([i[s:] for i, (s, _, _) in zip(ids, todo)]), device="cuda")
    pos = torch.as_tensor(np.concatenate([np.arange(s, s + n) for s, n, _ in todo]), device="cuda")
    ends = np.cumsum([n for _, n, _ in todo])
    sel = torch.as_tensor(np.concatenate([np.arange(e - s, e) for e, (_, _, s) in zip(ends, todo)]), device="cuda")

    def turn(x, at):
        a = f64(at)[:, None] * inv.cuda()[None, :]
        cos, sin = a.cos()[:, None, :], a.sin()[:, None, :]
        x = x.view(x.shape[0], -1, DIM)
        lo, hi = x[..., :DIM // 2], x[..., DIM // 2:]
        return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], -1)

    def attention(l, q, rows):
        out, at = [], 0
        for i, (cached, n, sampled) in enumerate(todo):
            r = n if rows else sampled
            total = cached + n
            k, v = (t[first[i]:first[i] + -(-total // BLOCK)].permute(0, 2, 1, 3).reshape(-1, KV_HEADS, DIM)[:total]
                    for t in cache[2 * l:2 * l + 2])
            out.append(attend(q[at:at + r], k, v, DIM ** -0.5))
            at += r
        return torch.cat(out)

    def store(l, k, v):
        at = 0
        for i, (cached, n, _) in enumerate(todo):
            p = torch.arange(cached, cached + n, device="cuda")
            for t, x in ((cache[2 * l], k), (cache[2 * l + 1], v)):
                t[first[i] + p // BLOCK, :, p % BLOCK] = x[at:at + n].view(n, KV_HEADS, DIM)
            at += n

    def mlp(x, b):
        x = rms(x, eps)
        g = torch.nn.functional.silu(lin(x, rnd(b + 5, FF, HIDDEN)))
        return lin(g * lin(x, rnd(b + 6, FF, HIDDEN)), rnd(b + 7, HIDDEN, FF))

    x, mine = f64(rnd(1, VOCAB, HIDDEN))[new], pos
    for l in range(c["layers"]):
        b, early = 100 + 20 * l, l < kv_layers(c)
        if not early and l == kv_layers(c):
            shared = rms(x, eps)
            for j in range(l, c["layers"]):
                bj = 100 + 20 * j
                store(j, turn(lin(shared, rnd(bj + 2, KV_HEADS * DIM, HIDDEN)), pos),
                      lin(shared, rnd(bj + 3, KV_HEADS * DIM, HIDDEN)))
            x, mine = x[sel], pos[sel]
        h = rms(x, eps)
        if early:
            store(l, turn(lin(h, rnd(b + 2, KV_HEADS * DIM, HIDDEN)), pos),
                  lin(h, rnd(b + 3, KV_HEADS * DIM, HIDDEN)))
        q = turn(lin(h, rnd(b + 1, HEADS * DIM, HIDDEN)), mine)
        x = x + lin(attention(l, q, early), rnd(b + 4, HIDDEN, HEADS * DIM))
        x = x + mlp(x, b)
    if not c["swiftkv"]:
        x = x[sel]
    return {"logits": rms(x, eps) @ f64(rnd(2, VOCAB, HIDDEN)).t(), "cache": cache}


def exact_taralix(c, seed):
    eps, rnd = 1e-6, Weights(seed).next
    todo, ids = spans(c), tokens_of(c, seed)
    first, blocks = blocks_of(c)
    W, H, D = T_WIDTH, T_HEADS, T_DIM
    cache = [torch.empty(blocks, 1, BLOCK, T_RANK, dtype=torch.bfloat16, device="cuda")
             for _ in range((c["layers"] + 1) // 2)]
    fill_cache(cache, seed)
    cache = [f64(t) for t in cache]
    # the checkpoint's order
    w = {"embed": rnd(VOCAB, W, std=1.0), "head": rnd(VOCAB, W), "final": rnd(W, std=0.1)}
    for i in range(c["layers"]):
        w["norm1", i], w["norm2", i] = rnd(W, std=0.1), rnd(W, std=0.1)
        w["q", i] = rnd(H * D, W)
        if i % 2 == 0:
            w["dkv", i] = rnd(T_RANK, W)
            w["ckv", i] = 1.0 + rnd(T_RANK, std=0.1)
        w["uk", i], w["uv", i], w["o", i] = rnd(H * D, T_RANK), rnd(H * D, T_RANK), rnd(W, H * D)
        w["router", i], w["bias", i] = rnd(T_EXPERTS, W), rnd(T_EXPERTS, std=0.1)
        for e in range(T_EXPERTS):
            w["expert", i, e] = rnd(T_FF, W), rnd(T_FF, W), rnd(W, T_FF)
    norm = lambda x, g: rms(x, eps) * (1.0 + f64(g))    # noqa: E731
    x = f64(w["embed"])[torch.as_tensor(np.concatenate([i[s:] for i, (s, _, _) in zip(ids, todo)]), device="cuda")]
    for i in range(c["layers"]):
        rows, at, out = cache[i // 2], 0, []
        if i % 2 == 0:
            latent = rms(x @ f64(w["dkv", i]).t(), eps) * f64(w["ckv", i])
        q = (x @ f64(w["q", i]).t()).view(-1, H, D)
        for j, (cached, n, _) in enumerate(todo):
            total = cached + n
            p = torch.arange(cached, total, device="cuda")
            if i % 2 == 0:
                rows[first[j] + p // BLOCK, 0, p % BLOCK] = latent[at:at + n]
            seen = rows[first[j]:first[j] + -(-total // BLOCK)].reshape(-1, T_RANK)[:total]
            out.append(attend(q[at:at + n], (seen @ f64(w["uk", i]).t()).view(total, H, D),
                              (seen @ f64(w["uv", i]).t()).view(total, H, D), D ** -0.5))
            at += n
        x = norm(T_ALPHA * x + torch.cat(out) @ f64(w["o", i]).t(), w["norm1", i])
        z, chosen = (x @ f64(w["router", i]).t() + f64(w["bias", i])).topk(T_TOP, -1)
        share, y = torch.softmax(z, -1), torch.zeros_like(x)
        for e in range(T_EXPERTS):
            t, k = torch.nonzero(chosen == e, as_tuple=True)
            g, u, d = (f64(m) for m in w["expert", i, e])
            y.index_add_(0, t, share[t, k, None] * ((torch.nn.functional.silu(x[t] @ g.t()) * (x[t] @ u.t())) @ d.t()))
        x = norm(T_ALPHA * x + y, w["norm2", i])
    ends = np.cumsum([n for _, n, _ in todo])
    sel = torch.as_tensor(np.concatenate([np.arange(e - s, e) for e, (_, _, s) in zip(ends, todo)]), device="cuda")
    return {"logits": norm(x[sel], w["final"]) @ f64(w["head"]).t(), "cache": cache}


def exact_fp8(c, seed):
    h, residual, weights = fp8_inputs(c, seed)
    h, residual = f64(h), f64(residual)
    for norm, gate_up, down in weights:
        residual = residual + h
        x = e4m3_rows(rms(residual, 1e-5) * f64(norm))
        g, u = (x @ e4m3(w).t() for w in gate_up.split(FF))
        h = e4m3_rows(torch.nn.functional.silu(g) * u) @ e4m3(down).t()
    return {"out": h, "residual": residual}


def exact_embed(c, seed):
    rnd, W, texts = Weights(seed), B_WIDTH, tokens_of(c, seed)
    lens = [len(t) for t in texts]
    ln = lambda x, b: torch.nn.functional.layer_norm(x, (W,), bias=f64(b), eps=1e-12)    # noqa: E731
    lin = lambda x, w, b: x @ f64(w).t() + f64(b)    # noqa: E731
    ids = torch.as_tensor(np.concatenate(texts), device="cuda")
    pos = torch.as_tensor(np.concatenate([np.arange(n) for n in lens]), device="cuda")
    x = f64(rnd(1, B_VOCAB, W))[ids] + f64(rnd(2, 512, W))[pos] + f64(rnd(3, 2, W))[0]
    x = ln(x, rnd(4, W))
    for l in range(B_LAYERS):
        b = 100 + 20 * l
        q, k, v = (lin(x, rnd(b + j, W, W), rnd(b + 3 + j, W)).view(-1, B_HEADS, W // B_HEADS) for j in range(3))
        out, at = [], 0
        for n in lens:
            out.append(attend(q[at:at + n], k[at:at + n], v[at:at + n], (W // B_HEADS) ** -0.5, False))
            at += n
        x = ln(x + lin(torch.cat(out), rnd(b + 6, W, W), rnd(b + 7, W)), rnd(b + 8, W))
        u = torch.nn.functional.gelu(lin(x, rnd(b + 9, B_FF, W), rnd(b + 10, B_FF)))
        x = ln(x + lin(u, rnd(b + 11, W, B_FF), rnd(b + 12, W)), rnd(b + 13, W))
    at = torch.as_tensor(np.cumsum([0] + lens[:-1]), device="cuda")
    return {"vectors": torch.nn.functional.normalize(x[at], dim=-1).cpu().numpy()}


def exact(case, seed):
    seed = seed % 100003
    with torch.inference_mode():
        return {"llama": exact_llama, "taralix": exact_taralix, "fp8": exact_fp8,
                "embed": exact_embed}[case["path"]](case, seed)
