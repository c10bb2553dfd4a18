"""The host-side planner of attention work items (``ops.plan_attention_work``)."""

import numpy as np
import pytest
import torch

from arcticinference_b200 import ops


def _covered(work, n_seq, kv_lens):
    """Every sequence's keys are covered exactly once by its work items."""
    got = {i: [] for i in range(n_seq)}
    for seq, tok, n, qpos, ks, ke, si, ns in work:
        if n > 0:
            got[int(seq)].append((int(ks), int(ke), int(si), int(ns)))
    for i, kl in enumerate(kv_lens):
        spans = sorted(got[i])
        assert spans[0][0] == 0 and spans[-1][1] >= kl
        for (a0, a1, _, _), (b0, _b1, _, _) in zip(spans, spans[1:]):
            assert a1 == b0
        assert all(ns == len(spans) for _, _, _, ns in spans)
        assert sorted(si for _, _, si, _ in spans) == list(range(len(spans)))


def test_tail_split_plan_cuts_the_last_round_only():
    # 128 sequences x 8 KV heads on 296 CTA slots: three full waves and 136 CTAs in a fourth;
    # the 17 sequences of that wave are cut in two so that their pieces cover the slots
    assert ops.tail_split_plan(128, 8, 296) == (17, 2)
    assert ops.tail_split_plan(64, 8, 296) == (0, 1)     # last wave 73 % full: left alone
    assert ops.tail_split_plan(37, 8, 296) == (0, 1)     # exactly one wave
    assert ops.tail_split_plan(16, 8, 296) == (0, 1)     # fewer CTAs than slots: other rule


def test_large_decode_batch_cuts_its_longest_sequences_and_places_the_pieces_last():
    kv = [2000 + i for i in range(128)]
    work, tok_splits, max_splits = ops.plan_attention_work([1] * 128, kv, 4, True, Hkv=8)
    assert max_splits == 2 and work.shape == (128 + 17, 8)
    assert sorted(np.nonzero(tok_splits == 2)[0].tolist()) == list(range(111, 128))
    _covered(work, 128, kv)
    lengths = work[:, 5] - work[:, 4]
    assert all(a >= b for a, b in zip(lengths, lengths[1:]))       # heaviest first
    assert set(work[-34:, 0].tolist()) == set(range(111, 128))      # the pieces come last
    # a cap of one split (a captured graph without partial buffers) is respected
    work, tok_splits, max_splits = ops.plan_attention_work([1] * 128, kv, 4, True, Hkv=8,
                                                           max_splits_cap=1)
    assert max_splits == 1 and work.shape[0] == 128


def test_small_decode_batch_is_split_to_occupy_the_gpu():
    kv = [4000] * 16
    work, tok_splits, max_splits = ops.plan_attention_work([1] * 16, kv, 4, True, Hkv=8)
    assert max_splits > 1
    _covered(work, 16, kv)
    assert np.all(work[:, 2] == 1)


def test_decode_splits_fill_at_most_two_waves():
    for ctas in (1, 8, 24, 64, 150, 192, 295):
        for tiles in (1, 4, 9, 24, 300):
            ns = ops.decode_splits(ctas, tiles, 296)
            assert 1 <= ns <= 16 and (ns == 1 or ctas * ns <= 592 and ns <= tiles // 2)
    assert ops.decode_splits(192, 24, 296) == 3


def test_captured_decode_plan_holds_every_mix_of_requests():
    rng = np.random.default_rng(0)
    for bucket in (1, 2, 8, 17, 32, 96, 128, 160):
        for hkv in (1, 8):
            plan = ops.DecodePlan(4, 4 * hkv, hkv, 128, bucket, 1, 64)
            for _ in range(40):
                n = int(rng.integers(1, bucket + 1))
                q = [1] * n if rng.random() < 0.5 else [4] * max(1, n // 4)
                q = q if sum(q) <= bucket else [1]
                kv = [int(k) for k in rng.integers(5, 9000, len(q))]
                if sum(q) < bucket:        # the padding tokens' own sequence
                    q, kv = q + [bucket - sum(q)], kv + [bucket - sum(q)]
                work, splits, most = plan.plan(q, kv)
                assert work.shape[0] <= plan.work_cap and most <= plan.splits
                _covered(work, len(q), kv) if max(q) == 1 else None


@pytest.mark.parametrize("block_size", [16, 64, 128])
@pytest.mark.parametrize("hkv,G,max_q", [(1, 4, 1), (2, 8, 1), (4, 8, 4), (8, 4, 1), (8, 4, 4), (8, 4, 16), (16, 1, 1),
                                         (1, 64, 1)])
def test_captured_decode_plan_holds_every_count_of_requests(block_size, hkv, G, max_q):
    """Whatever the cache's block size says about the kernel, the work list holds any number of requests, alone,
    with drafts, and with the padding tokens' sequence."""
    rng = np.random.default_rng(1)
    for bucket in (1, 4, 24, 56, 64, 96, 152, 304):
        plan = ops.DecodePlan(G, G * hkv, hkv, 128, bucket, max_q, block_size)
        host = np.zeros(plan.int32_words, dtype=np.int32)
        plan.bind(host, torch.zeros(plan.int32_words, dtype=torch.int32), None)
        for n in sorted({1, 2, bucket, *range(max(1, bucket - 16), bucket), *rng.integers(1, bucket + 1, 12).tolist()}):
            for q_lens in ([1] * n, [max_q] * max(1, n // max_q)):
                for kv in ([2000] * len(q_lens), rng.integers(max_q, 20000, len(q_lens)).tolist()):
                    q, kv = list(q_lens), list(kv)
                    if sum(q) > bucket:
                        continue
                    if sum(q) < bucket:
                        q, kv = q + [bucket - sum(q)], kv + [bucket - sum(q)]
                    work, splits, most = plan.plan(q, kv)
                    assert work.shape[0] <= plan.work_cap and most <= plan.splits, (bucket, n)
                    plan.fill(q, kv)


def test_plan_and_kernel_agree_on_the_ctas_that_an_sm_holds():
    """Blocks of 128 tokens take the kernel with one CTA per SM: pieces for 148 CTAs, not for 296."""
    for n in (1, 8, 18, 40):
        q, kv = [1] * n, [16384] * n
        m = {bs: ops.build_attention_metadata(q, kv, None, 4, 32, 128, "cpu", Hkv=8, block_size=bs) for bs in (64, 128)}
        assert m[64].tile_keys == 64 and m[128].tile_keys == 128
        for bs, meta in m.items():
            assert ops.DecodePlan(4, 32, 8, 128, n, 1, bs).tile_keys == meta.tile_keys
        if n * 8 < 148:
            assert m[128].num_work * 8 <= 148 and m[64].num_work >= m[128].num_work


def test_long_sequences_among_short_ones_are_cut_as_one_wave_allows():
    """However short the others are, no piece is longer than with as many pieces per sequence as one wave holds."""
    rng = np.random.default_rng(2)

    def longest(q_lens, kv, hkv, **kw):
        work, _, _ = ops.plan_attention_work(q_lens, kv, 4, True, Hkv=hkv, slots=296, **kw)
        _covered(work, len(kv), kv)
        return ((work[:, 5] - work[:, 4] + 127) // 128).max()

    cases = [([1] * n, [short] * (n - 1) + [32000], hkv) for n in (16, 24, 36) for hkv in (1, 2, 8) for short in (5, 900)]
    for _ in range(200):
        n, q = int(rng.integers(1, 38)), int(rng.choice([1, 4, 8]))
        cases.append(([q] * n, (2 ** rng.uniform(3, 15, n)).astype(int).tolist(), int(rng.choice([1, 2, 4, 8]))))
    for q_lens, kv, hkv in cases:
        assert longest(q_lens, kv, hkv, fill_slots=True) <= longest(q_lens, kv, hkv), (q_lens, kv, hkv)


# steps that were timed both ways, and by how much two tiles per CTA were the slower or the faster form
@pytest.mark.parametrize("q_lens,kv_lens,G,hkv,D,wide", [
    ([1474, 13], [1474, 84], 1, 16, 128, False),                                               # 1.17 times
    ([1] * 29 + [4, 384, 84, 160, 25, 116], [900] * 29 + [7, 6192, 86, 5315, 25, 159], 8, 2, 64, False),   # 1.21
    ([634, 3247], [634, 3247], 4, 2, 128, False), ([71, 4029], [71, 4029], 8, 1, 128, False),  # 1.23, 1.25
    ([2048] * 4, [2048] * 4, 4, 8, 128, True), ([3888], [3888], 4, 8, 128, True),              # 0.64, 0.57
    ([8192], [32768], 4, 8, 128, True), ([1] * 61 + [1987], [1500] * 61 + [1987], 4, 8, 128, True),        # 0.67, 0.88
    ([1] * 200, [2000] * 200, 4, 8, 128, False), ([], [], 4, 8, 128, False),
])
def test_two_tiles_of_rows_where_they_are_faster(q_lens, kv_lens, G, hkv, D, wide):
    assert ops.wide_tiles_pay(q_lens, kv_lens, G, hkv, D) == wide


def test_kernel_of_short_texts_within_a_wave():
    for longest, ctas, pays in ((1, 12, True), (64, 12, True), (65, 148, False), (128, 149, True), (129, 4000, False)):
        assert ops.short_attention_pays(longest, ctas) == pays
