"""Kernels on values that are no ordinary numbers, attention rows stored to several destinations, and whole steps with
and without programmatic launches."""

import ctypes
import math
import os
import subprocess
import sys

import pytest
import torch

from arcticinference_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEV) * scale).to(dtype)


def _cache(q_lens, kv_lens, Hq, Hkv, D, bs):
    torch.manual_seed(len(q_lens))
    blocks = [-(-k // bs) for k in kv_lens]
    bt, at = torch.zeros(len(q_lens), max(blocks), dtype=torch.int32), 1
    for i, n in enumerate(blocks):
        bt[i, :n] = torch.arange(at, at + n)
        at += n
    return _rand(sum(q_lens), Hq * D), _rand(at, Hkv, bs, D), _rand(at, Hkv, bs, D), bt.to(DEV)


def _attend(q, k, v, bt, q_lens, kv_lens, Hq, Hkv, D):
    """Causal attention in 64 bits."""
    out, at = [], 0
    for i, (n, kl) in enumerate(zip(q_lens, kv_lens)):
        rows = [c[bt[i].long()].transpose(1, 2).reshape(-1, Hkv, D)[:kl].double().transpose(0, 1) for c in (k, v)]
        kk, vv = (r.repeat_interleave(Hq // Hkv, 0) for r in rows)
        s = q[at:at + n].double().view(n, Hq, D).transpose(0, 1) @ kk.mT / math.sqrt(D)
        hidden = torch.arange(kl, device=DEV) > torch.arange(kl - n, kl, device=DEV)[:, None]
        w = torch.softmax(s.masked_fill(hidden, -math.inf), -1)
        out.append((w @ vv).transpose(0, 1).reshape(n, Hq * D))
        at += n
    return torch.cat(out)


def _same(got, want, rel=2e-2):
    assert torch.equal(got.isnan(), want.isnan())
    ok = want.isnan() | ((got.double() - want).abs() <= rel * (1 + want.abs()))
    assert ok.all()


# (probabilities and results in bf16, 2^-8 of the value each, over values of size 1)
@pytest.mark.parametrize("wide", [True, False])
@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf])
def test_paged_attention_of_odd_keys(value, wide, monkeypatch):
    """One number of one key is none: rows that see the key have no result, or one without it; rows before it and other
    sequences are as ever. Two tiles of rows per CTA and one."""
    monkeypatch.setattr(ops, "wide_tiles_pay", lambda *a: wide)
    q_lens, kv_lens, Hq, Hkv, D, bs = [300, 40], [450, 40], 4, 2, 128, 32
    q, k, v, bt = _cache(q_lens, kv_lens, Hq, Hkv, D, bs)
    k[bt[0, 200 // bs].long(), 1, 200 % bs, 7] = value
    meta = ops.build_attention_metadata(q_lens, kv_lens, bt, 2, Hq, D, DEV, Hkv=Hkv, wide=True, allow_split=False)
    assert (meta.tile_keys == ops.WIDE_ROWS) == wide
    out = ops.attention(q, k, v, meta, Hq, Hkv, D)
    ops.check_status()
    want = _attend(q, k, v, bt, q_lens, kv_lens, Hq, Hkv, D)
    assert want.isnan().any() and not want.isnan().all()
    _same(out, want)


@pytest.mark.parametrize("wide", [True, False])
def test_paged_attention_of_equal_low_scores(wide, monkeypatch):
    """Scores far below zero weigh by their differences: equal ones give the mean."""
    monkeypatch.setattr(ops, "wide_tiles_pay", lambda *a: wide)
    q_lens, kv_lens, Hq, Hkv, D, bs = [300], [300], 2, 2, 64, 64
    q, k, v, bt = _cache(q_lens, kv_lens, Hq, Hkv, D, bs)
    q.zero_()
    k.zero_()
    q[:, ::D], k[..., 0] = 2.0 ** 5, -2.0 ** 6
    meta = ops.build_attention_metadata(q_lens, kv_lens, bt, 1, Hq, D, DEV, Hkv=Hkv, wide=True, allow_split=False)
    out = ops.attention(q, k, v, meta, Hq, Hkv, D)
    ops.check_status()
    _same(out, _attend(q, k, v, bt, q_lens, kv_lens, Hq, Hkv, D))


@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf])
def test_encoder_attention_short_of_odd_keys(value, monkeypatch):
    monkeypatch.setattr(ops, "short_attention_pays", lambda longest, ctas: True)
    H, D, lens = 2, 64, [70, 33, 128]
    qkv = _rand(sum(lens), 3 * H * D)
    qkv[80, H * D + 3] = value      # a key of the second sequence, first head
    out = ops.attention_contiguous(qkv[:, :H * D], qkv[:, H * D:2 * H * D], qkv[:, 2 * H * D:], lens, H, D)
    ops.check_status()
    want, at = [], 0
    for n in lens:
        q, k, v = (t.double() for t in qkv[at:at + n].view(n, 3, H, D).permute(1, 2, 0, 3))
        want.append((torch.softmax(q @ k.mT / math.sqrt(D), -1) @ v).transpose(0, 1).reshape(n, H * D))
        at += n
    _same(out, torch.cat(want))


def test_linear_silu_of_odd_rows():
    """Rows with an infinity or none at all: gate and up of either sign, silu(-inf) has no value."""
    M, inter, K = 300, 128, 64
    x, w = _rand(M, K), _rand(2 * inter, K, scale=0.2)
    x[3, 5], x[7, 0], x[260, 1] = math.inf, math.nan, -math.inf
    out = ops.linear_silu(x, w)
    ops.check_status()
    z = x.double() @ w.double().t()
    g, u = z[:, :inter], z[:, inter:]
    want = g * torch.sigmoid(g) * u
    inf = want.isinf()
    assert inf[3].any() and inf[260].any() and want[7].isnan().all()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.double()[inf], want[inf])
    ok = inf | want.isnan() | ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-4)
    assert ok.all()


# keys in one piece and cut, so that the fold stores the rows
@pytest.mark.parametrize("D,split", [(128, False), (64, False), (128, True)])
def test_wide_attention_to_local_destinations(D, split, monkeypatch):
    """Both destinations in this GPU's memory: rows t of the first half in buffer 0, of the second in buffer 1, the
    heads behind those of an earlier rank."""
    monkeypatch.setattr(ops, "wide_tiles_pay", lambda *a: True)
    from arcticinference_b200.ops import native
    q_lens, kv_lens, Hq, Hkv, bs, world = [129, 95], [1300, 95], 4, 2, 64, 2
    T, n = sum(q_lens), sum(q_lens) // world
    q, k, v, bt = _cache(q_lens, kv_lens, Hq, Hkv, D, bs)
    meta = ops.build_attention_metadata(q_lens, kv_lens, bt, 2, Hq, D, DEV, Hkv=Hkv, wide=True, allow_split=split)
    assert meta.tile_keys == ops.WIDE_ROWS and (meta.max_splits > 1) == split
    cols = world * Hq * D
    bufs = [torch.zeros(n + 3, cols, dtype=torch.bfloat16, device=DEV) for _ in range(world)]
    ptrs = (ctypes.c_void_p * world)(*[b.data_ptr() + Hq * D * 2 for b in bufs])
    P, I, LL, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    native.declare("ab200_attention_scatter", I, [P, LL, P, P, LL, I, P, I, P, I, P, I, LL, I, I, I, F, P, I, I, LL, P, P,
                                                  I, P, P])
    rc = native.lib().ab200_attention_scatter(
        q.data_ptr(), q.stride(0), k.data_ptr(), v.data_ptr(), k.shape[0], bs, bt.data_ptr(), bt.shape[1],
        meta.work.data_ptr(), meta.num_work, native.ptr(meta.tok_splits), meta.max_splits, T, Hq, Hkv, D,
        1 / math.sqrt(D), ptrs, world, n, cols, native.ptr(meta.o_part), native.ptr(meta.lse_part), meta.tile_keys,
        native.status_buffer(q.device).data_ptr(), native.stream_ptr())
    assert rc == 0
    ops.check_status()
    want = _attend(q, k, v, bt, q_lens, kv_lens, Hq, Hkv, D)
    for j, b in enumerate(bufs):
        _same(b[:n, Hq * D:], want[j * n:(j + 1) * n])
        assert not b[n:].any() and not b[:, :Hq * D].any()


CHILD = '''
import dataclasses, sys
import numpy as np, torch
from arcticinference_b200 import ops
from arcticinference_b200.config import (PRESETS, CacheConfig, EngineConfig, ParallelConfig, SchedulerConfig)
from arcticinference_b200.embedding.engine import EmbeddingEngine
from arcticinference_b200.engine.llm_engine import LLMEngine
from arcticinference_b200.engine.request import Request
from arcticinference_b200.engine.sampling_params import SamplingParams
from arcticinference_b200.engine.scheduler import ScheduledRequest, SchedulerOutput
from arcticinference_b200.ops import stream_ops as st

out, rng = {}, np.random.default_rng(0)
enc = EmbeddingEngine("bert-tiny", device="cuda:0", max_num_batched_tokens=1024, max_num_seqs=64)
for name, most in (("short", 60), ("long", 500)):
    texts = [rng.integers(0, 1000, int(n)) for n in rng.integers(1, most, 24)]
    out["encoder " + name] = torch.from_numpy(enc.encode(texts))

for quant in (None, "fp8"):
    model = dataclasses.replace(PRESETS["llama-small"], quantization=quant)
    engine = LLMEngine(EngineConfig(model=model, parallel=ParallelConfig(),
                                    cache=CacheConfig(block_size=64, num_gpu_blocks=96, enable_prefix_caching=False),
                                    scheduler=SchedulerConfig(max_model_len=1024, max_num_seqs=64),
                                    load_format="dummy", seed=0), device="cuda")
    reqs = []
    for i, n in enumerate((700, 301, 5, 64)):
        r = Request("r%d" % i, rng.integers(0, 32000, n + 8).tolist(), SamplingParams(temperature=0.0, ignore_eos=True))
        r.block_ids = list(range(1 + 16 * i, 17 + 16 * i))
        reqs.append((r, n))
    with torch.inference_mode():
        for t in range(4):        # a prompt step, then captured one-token steps
            step = SchedulerOutput()
            for r, n in reqs:
                at, new = (0, n) if t == 0 else (n + t - 1, 1)
                step.scheduled.append(ScheduledRequest(r, at, new, 0, True, want=[new - 1]))
                step.total_tokens += new
            out["%s step %d" % (quant, t)] = engine.runner.score(step).cpu()
    assert engine.runner.graph_replays >= 3
    del engine

gen = torch.Generator(device="cuda").manual_seed(0)
rand = lambda *s: torch.randn(*s, device="cuda", generator=gen)
x, w, b = rand(3001, 256).bfloat16(), rand(6, 256) * 0.1, torch.zeros(6, device="cuda")
w1, w2 = (rand(6, 1024, 256) / 16).bfloat16(), (rand(6, 256, 512) / 22).bfloat16()
r, rows = st.route(x, x, w.bfloat16(), b, 3)
assert r.even
y = st.grouped_linear(st.grouped_linear(rows, w1, r, act="silu"), w2, r)
out["experts"] = y[r.rows.long()].cpu()        # (the order within an expert is free)
ops.check_status()
torch.save(out, sys.argv[1])
'''


def test_programmatic_launches_change_no_bit(tmp_path):
    """AB200_PDL moves the start of kernels and nothing else: embeddings of short and long texts, a prompt step and
    captured decode steps of a bf16 and an fp8 model, and experts on pairs of tiles are equal in every bit, so
    nothing reads an input or a weight too early."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    got = []
    for i, flag in enumerate("101"):
        env = dict(os.environ, AB200_PDL=flag, ARCTIC_B200_NO_AUTOBUILD="1", PYTHONPATH=root)
        path = str(tmp_path / str(i))
        run = subprocess.run([sys.executable, "-c", CHILD, path], env=env, capture_output=True, text=True, timeout=600)
        assert run.returncode == 0, run.stderr[-3000:]
        got.append(torch.load(path))
    for other in got[1:]:
        assert got[0].keys() == other.keys() and len(other) == 11
        assert not [k for k in other if not torch.equal(got[0][k], other[k])]
