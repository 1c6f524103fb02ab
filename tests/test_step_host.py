"""Host-side decisions of the step function that need no device: the list of query tiles a step
hands to the prompt attention kernel, and the shape a step of many tokens is captured for."""

from __future__ import annotations

import random
from types import SimpleNamespace

import numpy as np

from kvforge_b200.engine.step import BatchItem, ModelRunner, _Layout


def layout_with(q_lens, ctx_lens, tile_sizes, n_cap=None, b_cap=None):
    nb = len(q_lens)
    lay = _Layout(n_cap or sum(q_lens), b_cap or nb, 4, 1, nb, tuple(tile_sizes))
    host = np.zeros(lay.total, dtype=np.int32)
    host[lay.off["qsl"] : lay.off["qsl"] + nb + 1] = np.concatenate([[0], np.cumsum(q_lens)])
    host[lay.off["ctx"] : lay.off["ctx"] + nb] = ctx_lens
    return lay, host


def test_query_tiles_cover_every_query_once_longest_walk_first():
    rng = random.Random(4)
    for _ in range(50):
        nb = rng.randint(1, 9)
        q_lens = [rng.choice([1, 1, 2, 5, 31, 32, 33, 100]) for _ in range(nb)]
        ctx_lens = [q + rng.randint(0, 300) for q in q_lens]
        sizes = rng.sample([1, 16, 32, 64, 128], 2)
        lay, host = layout_with(q_lens, ctx_lens, sizes, n_cap=sum(q_lens) + rng.randint(0, 70), b_cap=nb + rng.randint(0, 3))
        counts = ModelRunner._fill_query_tiles(None, host, lay, nb)
        for tq in lay.tile_sizes:
            cap = lay.tile_cap(tq)
            total, n_multi, n_single = counts[tq]
            assert n_single == sum(1 for q in q_lens if q == 1)
            assert total == sum(-(-q // tq) for q in q_lens) <= cap
            for name, n_live, wanted in ((f"qtiles_{tq}", total, q_lens), (f"qtiles_multi_{tq}", n_multi, [q if q > 1 else 0 for q in q_lens])):
                tiles = host[lay.off[name] : lay.off[name] + 2 * cap].reshape(cap, 2)
                assert (tiles[n_live:, 0] == -1).all()
                seen = [set() for _ in range(nb)]
                last_keys = []
                for seq, q0 in tiles[:n_live]:
                    assert q0 % tq == 0 and 0 <= q0 < wanted[seq]
                    assert q0 not in seen[seq]
                    seen[seq].add(int(q0))
                    last_keys.append(ctx_lens[seq] - q_lens[seq] + min(q_lens[seq], q0 + tq))
                assert [len(s) for s in seen] == [-(-w // tq) for w in wanted]
                assert last_keys == sorted(last_keys, reverse=True)


def test_the_shape_a_step_is_captured_for():
    runner = SimpleNamespace(max_model_len=8192)
    items = [BatchItem("a", [1] * 700, 300, "last"), BatchItem("b", [5], 2000, "last")]
    # contexts up to 2,001 tokens: graphs reach the next power of two; a single token is among the sequences
    assert ModelRunner._graph_key(runner, items, 704, 2, False) == (704, 2, 2048, True, False)
    assert ModelRunner._graph_key(runner, items[:1], 704, 1, False) == (704, 1, 1024, False, False)
    # the decode form (one token per sequence) has no such distinction
    assert ModelRunner._graph_key(runner, [BatchItem("b", [5], 5000, "last")], 1, 1, True) == (1, 1, 8192, False, True)
    runner.max_model_len = 4096
    assert ModelRunner._graph_key(runner, [BatchItem("b", [5], 4000, "last")], 1, 1, True)[2] == 4096


def test_a_step_of_many_tokens_padded_to_its_sequence_count_is_no_decode_graph():
    """64 tokens in 64 sequences come two ways: 64 decoding requests (the decode form), or some
    decoding requests beside a short portion of a prompt, padded to 64 and 64.  The two are
    different graphs (the second computes every query of the portion) and must not share a key."""
    runner = SimpleNamespace(max_model_len=4096)
    decoding = [BatchItem(f"d{i}", [3], 100 + i, "last") for i in range(64)]
    mixed = [BatchItem(f"d{i}", [3], 100 + i, "last") for i in range(40)] + [BatchItem("p", [1] * 20, 0, "last")]
    a = ModelRunner._graph_key(runner, decoding, 64, 64, True)
    b = ModelRunner._graph_key(runner, mixed, 64, 64, False)
    assert a != b and a[:3] == b[:3]


def test_when_the_library_product_is_cut_into_slices_of_k():
    from kvforge_b200 import ops

    # a few dozen tokens, an output no wider than K, K of 2,048 or more: 4 slices up to 64 rows, 2 up to 128
    assert ops.library_splits(17, 2048, 2048) == 4 and ops.library_splits(64, 2048, 8192) == 4
    assert ops.library_splits(65, 4096, 14336) == 2 and ops.library_splits(128, 3072, 3072) == 2
    # the decode GEMM's rows, many rows, a wide output, a short K: the plain product
    assert ops.library_splits(16, 2048, 2048) == 1 and ops.library_splits(129, 2048, 8192) == 1
    assert ops.library_splits(32, 16384, 2048) == 1 and ops.library_splits(32, 96, 160) == 1
    assert ops.library_splits(32, 2048, 2048 + 64) == 1  # K that does not cut into 4 slices of whole 64s


def test_slices_of_the_decode_product_and_ranges_of_the_decode_attention():
    import random

    from kvforge_b200 import ops

    # the 1B shape: qkv / output / down up to 8 tokens, and from 9 on
    assert [ops.skinny_splits(n, k, 8) for n, k in ((3072, 2048), (2048, 2048), (2048, 8192))] == [8, 8, 10]
    assert [ops.skinny_splits(n, k, 16) for n, k in ((3072, 2048), (2048, 2048), (2048, 8192))] == [5, 8, 8]
    assert ops.skinny_splits(16384, 2048, 8) == 1 and ops.skinny_splits(96, 128, 4) == 1
    # no slice is ever empty: the kernel cuts K into slices of whole 64s, the same number of them each but the last
    rng = random.Random(0)
    for _ in range(2000):
        n, k, m = rng.randrange(8, 20000), 8 * rng.randrange(1, 2500), rng.choice((1, 8, 9, 16))
        s = ops.skinny_splits(n, k, m)
        per = -(-(-(-k // 64)) // s) * 64
        assert 1 <= s <= ops.SKINNY_MAX_SPLIT and (s - 1) * per < k, (n, k, m, s)
    # key ranges: 128 with 17 to 64 (sequence, kv head) pairs, 512 from 256 on, else 256; one size for one sequence
    sizes = {pairs: ops.attention_split_size(pairs, 1, 4096) for pairs in (1, 8, 16, 17, 64, 65, 255, 256, 2048)}
    assert sizes == {1: 256, 8: 256, 16: 256, 17: 128, 64: 128, 65: 256, 255: 256, 256: 512, 2048: 512}
    assert ops.ATTN_MIN_SPLIT == min(sizes.values())
    assert ops.attention_split_size(64, 1, 1 << 17, reach=4096) == 128 and ops.attention_split_size(64, 1, 1 << 17, reach=8192) == 256
    # heads wider than 64: a CTA holds twice the bytes, so short ranges only up to 32 pairs and half the CTAs a wave
    assert ops.attention_split_size(8, 8, 4096, 4096, head_dim=128) == 256 and ops.attention_split_size(4, 8, 4096, 4096, head_dim=128) == 128
    assert ops.attention_wave_target(8, 8, 64) == 888 and ops.attention_wave_target(8, 8, 128) == 444 and ops.attention_wave_target(64, 8, 128) == 3072
    # and never more ranges than the merge takes
    assert -(-(1 << 20) // ops.attention_split_size(8, 8, 1 << 20)) <= ops.MAX_ATTN_SPLITS


def test_a_step_of_single_tokens_is_laid_out_as_its_tables_say():
    """The arrays of a step whose requests bring one token each, against the block manager's lists: full, window and
    chunk groups whose pages have grown and come back, tokens from the host and from the device, a padded layout."""
    import pytest
    import torch

    from kvforge_b200.cache.block_manager import BlockManager, GroupSpec
    from kvforge_b200.cache.state_slots import StateSlotPool

    rng = random.Random(9)
    for case in range(20):
        bs = rng.choice([4, 16, 24])
        bm = BlockManager(400, bs, 0.0, [GroupSpec(), GroupSpec("window", 40, rng.choice([0, 9])), GroupSpec("chunk", 48)])
        runner = object.__new__(ModelRunner)
        runner.block_manager, runner.block_size, runner._copy_done, runner.n_groups = bm, bs, None, 3
        runner.max_model_len, runner.state_slots, runner.token_feedback = 300, StateSlotPool(8), object()
        items = []
        for i in range(rng.randint(1, 6)):
            start = rng.randint(0, 250)
            bm.allocate(f"r{i}", 1, 1)
            for at in range(0, start + 1, 7):
                bm.append_slots(f"r{i}", min(at + 7, start + 1), at)
            if rng.random() < 0.7:
                runner.state_slots.allocate(f"r{i}")
            wanted = rng.choice(["last", "all", "none", [0]])
            items.append(BatchItem(f"r{i}", [rng.randrange(1000)], start, wanted, feedback_row=rng.choice([None, 3])))
        bm.check_invariants()
        nb = len(items)
        cap = nb + rng.randint(0, 3)
        lay = _Layout(cap, cap, 80, 3, cap)
        runner._host = torch.full((lay.total,), 7, dtype=torch.int32)
        n, b, r, max_q, max_ctx = runner._fill(items, lay, padded=True, tiles=False)
        host, o = runner._host.numpy(), lay.off
        view = lambda name, size: host[o[name] : o[name] + size].tolist()  # noqa: E731
        rows = [i for i, it in enumerate(items) if it.wanted()]
        assert (n, b, r, max_q, max_ctx) == (nb, nb, len(rows), 1, max(it.start_pos for it in items) + 1)
        assert view("token_ids", cap) == [0 if it.feedback_row is not None else it.token_ids[0] for it in items] + [0] * (cap - nb)
        assert view("feedback_rows", cap) == [-1 if it.feedback_row is None else 3 for it in items] + [-1] * (cap - nb)
        assert view("positions", nb) == [it.start_pos for it in items]
        assert view("ctx", cap) == [it.start_pos + 1 for it in items] + [0] * (cap - nb)
        assert view("qsl", cap + 1) == [min(i, nb) for i in range(cap + 1)]
        assert view("logit_rows", r) == rows
        assert view("state_slots", cap) == [runner.state_slots.slot(it.seq_id) if runner.state_slots.has(it.seq_id) else -1 for it in items] + [-1] * (cap - nb)
        for g in range(3):
            at = o["slots"] + g * cap
            assert host[at : at + cap].tolist() == [bm.slots(it.seq_id, it.start_pos, it.start_pos + 1, g)[0] for it in items] + [-1] * (cap - nb)
            for i, it in enumerate(items):
                used = it.start_pos // bs + 1
                at = o["tables"] + (g * cap + i) * 80
                assert host[at : at + used].tolist() == bm.get_block_table(it.seq_id, g)[:used]
        with pytest.raises(ValueError):
            runner._fill([BatchItem("r0", [1], 300, "last")], lay)
        with pytest.raises(RuntimeError):  # the token's page was given back
            bm.allocate("gone", 1, 1)
            bm.append_slots("gone", 250, 249)
            runner._fill([BatchItem("gone", [1], 20, "last")], lay)


def test_pages_taken_at_once_are_those_taken_one_by_one():
    """Tables of full, window and chunk groups under random growth, and their arrays, against a manager that takes every page by
    itself and keeps lists alone."""
    import numpy as np
    import pytest

    from kvforge_b200.cache.block_manager import RELEASED, BlockManager, GroupSpec, NoFreeBlocksError

    class OneByOne:
        def __init__(self, n):
            self.free, self.tables = list(range(n - 1, -1, -1)), {}

        def allocate(self, seq, pages):
            self.tables[seq] = [self.free.pop() for _ in range(pages)]

        def append(self, seq, want, first, kept):
            table = self.tables[seq]
            for i in range(kept, min(first, len(table))):
                if table[i] >= 0:
                    self.free.append(table[i])
                    table[i] = RELEASED
            while len(table) < want:
                table.append(RELEASED if kept <= len(table) < first else self.free.pop())
            for i in [*range(min(kept, want)), *range(first, want)]:
                if table[i] < 0:
                    table[i] = self.free.pop()

        def release(self, seq):
            self.free += [b for b in reversed(self.tables.pop(seq)) if b >= 0]

    rng = random.Random(3)
    for case in range(10):
        bs = rng.choice([1, 4, 16])
        specs = [GroupSpec(), GroupSpec("window", 40, rng.choice([0, 9])), GroupSpec("chunk", 48)]
        bm, plain = BlockManager(900, bs, 0.0, specs), [OneByOne(900) for _ in specs]
        at = {}
        for step in range(200):
            seq = f"r{rng.randrange(5)}"
            if seq not in at:
                n, scheduled = rng.randint(1, 60), rng.choice([1, 7, 30])
                bm.allocate(seq, n, scheduled)
                for g, p in enumerate(plain):
                    p.allocate(seq, -(-(n if g == 0 else min(n, scheduled)) // bs))
                at[seq] = 0
            elif at[seq] > 120 or rng.random() < 0.1:
                bm.free(seq)
                for p in plain:
                    p.release(seq)
                del at[seq]
            else:
                start = max(0, at[seq] - rng.choice([0, 0, 0, 13]))  # sometimes back: pages that came back are taken anew
                end = start + rng.choice([1, 1, 5, 33])
                bm.append_slots(seq, end, start)
                for g, (p, spec) in enumerate(zip(plain, specs)):
                    first = 0 if g == 0 else max(0, start - 39) // bs if g == 1 else (start - start % 48) // bs
                    p.append(seq, -(-end // bs), first, min(-(-spec.keep_first // bs), first) if g else 0)
                at[seq] = end
            bm.check_invariants()
            for g, p in enumerate(plain):
                for s in at:
                    assert bm.get_block_table(s, g) == p.tables[s] and np.array_equal(bm.table_array(s, g), p.tables[s]), (case, step, g, s)
    pool = BlockManager(5, 4)._pools[0]
    assert pool.take(0) == [] and pool.take(-2) == [] and pool.take(3) == [0, 1, 2] and pool.pop() == 3
    with pytest.raises(NoFreeBlocksError):
        pool.take(2)
    assert pool.take(1) == [4] and pool.held == [True] * 5


def test_buffers_of_the_delta_rule_s_walk_hold_what_the_walk_may_see():
    """Where steps of more than four tokens a sequence go in groups, the walk's buffers are made for four tokens a sequence."""
    from types import SimpleNamespace

    import torch

    from kvforge_b200 import PRESETS
    from kvforge_b200.engine.core import spec_from_config
    from kvforge_b200.parts.base import PartSpec, build_part

    spec = next(p for s in spec_from_config(PRESETS["mopilorn-1b"]).layers for p in [s.block.params["mixer"]] if p.kind == "gated_delta_rule")
    for dtype, dk, budget, seqs, want in (
        (torch.bfloat16, 128, 2048, 64, (True, 256)), (torch.bfloat16, 128, 2048, 1000, (True, 2048)), (torch.bfloat16, 65, 512, 3, (True, 12)),
        (torch.bfloat16, 64, 2048, 64, (False, 2048)), (torch.bfloat16, 256, 2048, 64, (False, 2048)), (torch.float32, 128, 2048, 64, (False, 2048)),
    ):  # fmt: skip
        part = build_part("mixer", PartSpec(spec.kind, {**spec.params, "head_dim": dk}), "")
        part.rt = SimpleNamespace(dtype=dtype, max_tokens=budget, max_seqs=seqs)
        assert part._walk_rows(1) == want, (dtype, dk)
        assert part._walk_rows(2000) == (want[0], budget)


def test_buffer_of_the_delta_rule_s_chunks_follows_the_rule_and_not_the_request_slots():
    from types import SimpleNamespace

    import torch

    from kvforge_b200 import PRESETS, ops
    from kvforge_b200.engine.core import spec_from_config
    from kvforge_b200.parts.base import build_part

    for model in ("mopilorn-1b", "mopilorn-3b"):
        for layer in spec_from_config(PRESETS[model]).layers:
            if layer.block.params["mixer"].kind != "gated_delta_rule":
                continue
            part, asked = build_part("mixer", layer.block.params["mixer"], ""), []
            for budget, slots in ((2048, 256), (2048, 1), (700, 64), (400, 8)):
                part.rt = SimpleNamespace(max_tokens=budget, max_seqs=slots, buf=lambda name, rows, cols, dtype, cap: asked.append((rows, cols, cap)))
                widest = 0
                for n in range(1, budget + 1):
                    for seqs in range(1, slots + 1):
                        if ops.delta_chunks_ok(torch.bfloat16, part.dk, part.dv, part.H, part.decay == "channel", n, seqs, n):
                            if n in (384, 1000, budget):
                                part._chunks(n, seqs)
                                assert asked[-1][0] <= asked[-1][2] and asked[-1][0] * asked[-1][1] == ops.delta_chunk_floats(n, seqs, part.H, part.dv)
                            widest = max(widest, n // ops.DELTA_CHUNK_TOKENS + seqs)
                assert widest <= asked[-1][2] <= budget // 64 + budget // 96  # no record that no step can use, whatever the slots


def test_steps_that_go_in_chunks_are_those_measured_faster():
    """Groups of four against chunks of sixty-four, heads of 128 x 128: (heads, a decay a channel, lengths, chunks are faster)."""
    import torch

    from kvforge_b200 import ops

    for heads, channel, lens, faster in (
        (4, True, [256] * 2, False), (8, True, [256], False), (8, True, [256] * 2, True), (16, True, [256], True), (32, True, [256], True), (4, True, [384], True),
        (16, True, [1000] + [1] * 8, True), (16, True, [400] + [1] * 20, False), (32, True, [500] + [1] * 3, False), (24, True, [500] + [1] * 3, True), (16, True, [64] * 30, False),
        (8, False, [256], False), (8, False, [256] * 2, False), (16, False, [256] * 2, True), (32, False, [256], True), (4, False, [384], True), (8, False, [64] * 30, False),
        (24, False, [1000] + [1] * 8, False), (32, False, [500] + [1] * 3, False), (16, False, [700] + [100] * 6, True), (24, False, [500] * 4, True),
    ):  # fmt: skip
        assert ops.delta_chunks_ok(torch.bfloat16, 128, 128, heads, channel, sum(lens), len(lens), max(lens)) == faster, (heads, channel, lens)
    assert not ops.delta_chunks_ok(torch.float32, 128, 128, 16, True, 2048, 1, 2048) and not ops.delta_chunks_ok(torch.bfloat16, 64, 128, 16, True, 2048, 1, 2048)


def test_shaped_scores_keep_the_ranges_of_the_launch(monkeypatch):
    """The decode kernel may lengthen its ranges for plain scores in bfloat16 alone, in steps of single tokens and in mixed ones."""
    from types import SimpleNamespace

    import torch

    from kvforge_b200 import ops
    from kvforge_b200.parts.attention import PagedAttention

    calls = []
    monkeypatch.setattr(ops, "paged_attention", lambda *a, **kw: calls.append(kw))
    for dtype, shape, lengthens in (
        (torch.bfloat16, {}, True), (torch.bfloat16, {"sinks": object()}, True), (torch.float32, {}, False),
        (torch.bfloat16, {"bias": object()}, False), (torch.bfloat16, {"keep_first": 4}, False), (torch.bfloat16, {"softcap": 30.0}, False),
    ):  # fmt: skip
        part = object.__new__(PagedAttention)
        for k, v in dict(window=64, chunk=None, dv=64, keep_first=0, bias=None, softcap=0.0, sinks=None, nh=8, nkv=2, d=64, scale=0.1, _query_tile=32).items():
            setattr(part, k, shape.get(k, v))
        part.rt = SimpleNamespace(err=None, capturing=False)
        part._scratch = lambda ctx: ((), 100, 64)
        q, cache = torch.zeros(8, 512, dtype=dtype), SimpleNamespace(k=torch.zeros(4, 2, 16, 64), v=None, group=0)
        tiles = SimpleNamespace(num_single=3, multi=None, multi_count=1, tiles=None, count=4)
        for single in (True, False):
            calls.clear()
            ctx = SimpleNamespace(
                block_tables=[None], query_start_loc=None, context_lens=None, num_seqs=4, max_query_len=1 if single else 9, block_size=16,
                all_single_query=single, query_tiles={} if single else {32: tiles}, context_bound=0, max_context_len=50,
            )  # fmt: skip
            part.attend(ctx, q, 512, None, cache)
            ranges = [kw for kw in calls if kw.get("scratch") is not None]
            assert len(ranges) == (1 if single or dtype == torch.bfloat16 else 0)
            assert all((kw["wave_target"] > 0) == lengthens for kw in ranges), shape


def test_kernel_of_shaped_scores_by_the_times_of_both():
    """Steps of many sequences, few tokens, short and long contexts: (head size, heads a key head, key heads, sequences, tokens each,
    longest context, with a bias, us on the mma.sync kernel, us on the tcgen05 kernel), as timed.  The chosen kernel takes at most
    a tenth more than the mma.sync kernel and at most a fifth more than the better of the two."""
    from kvforge_b200 import ops

    timed = [
        (64, 4, 8, 1, 2, 2, True, 5.5, 9.8), (64, 4, 8, 1, 64, 64, True, 8.2, 10.0), (64, 4, 8, 1, 128, 128, True, 11.2, 10.6),
        (64, 4, 8, 1, 256, 256, True, 17.6, 15.1), (64, 4, 8, 40, 2, 384, True, 38.3, 39.9), (64, 4, 8, 40, 32, 192, True, 31.4, 28.2),
        (64, 4, 8, 40, 40, 40, True, 19.8, 28.3), (64, 4, 8, 8, 192, 192, True, 28.4, 23.7), (64, 4, 8, 4, 2, 256, True, 25.7, 15.8),
        (64, 8, 4, 8, 32, 256, True, 18.3, 15.4), (64, 8, 4, 1, 32, 192, True, 14.7, 14.3), (64, 8, 4, 8, 2, 80, True, 9.6, 11.2),
        (64, 1, 16, 20, 32, 80, False, 10.9, 21.0), (64, 1, 16, 40, 32, 384, False, 43.5, 60.4), (64, 1, 16, 4, 384, 384, False, 25.0, 19.8),
        (128, 3, 8, 20, 2, 80, False, 14.1, 25.8), (128, 3, 8, 40, 32, 64, False, 28.5, 33.4), (128, 3, 8, 4, 384, 384, False, 88.7, 47.6),
        (128, 3, 8, 4, 2, 192, False, 21.6, 17.5), (128, 4, 4, 1, 2, 256, True, 35.9, 20.6), (128, 4, 4, 4, 32, 128, True, 17.7, 13.6),
        (128, 4, 4, 20, 40, 40, True, 12.0, 23.6), (128, 4, 4, 20, 2, 384, True, 56.5, 24.8), (64, 4, 8, 1, 2048, 2048, True, 148.9, 76.2),
    ]  # fmt: skip
    for d, g, nkv, seqs, n, keys, biased, mma, tcgen05 in timed:
        took = tcgen05 if ops.shaped_tcgen05_pays(d, g, nkv, seqs, seqs * n, n, keys, biased) else mma
        assert took <= 1.1 * mma and took <= 1.2 * min(mma, tcgen05), (d, g, seqs, n, keys, took)
    assert ops.shaped_tcgen05_pays(64, 4, 8, 2, 2048, 1536, 2048, True) and ops.shaped_tcgen05_pays(64, 128, 1, 1, 40, 40, 4096, False)
