"""Host-side bounds that size kernel launches: they must never be below what the kernels will need (no GPU)."""
import random

import pytest

from sharpinference_b200.kernels import ops


def visible_lo(pos: int, kind: int, span: int) -> int:
    """First visible key of a row at ``pos``: the mask rule of csrc/common.cuh, restated."""
    if kind == ops.MASK_CHUNK:
        return pos // span * span
    if kind == ops.MASK_WINDOW:
        return max(0, pos - span + 1)
    return 0


def splits_of(pos: int, kind: int, span: int) -> int:
    """The 256-key splits (at absolute multiples of 256) that hold a visible key of the row."""
    return pos // ops.DECODE_SPLIT - visible_lo(pos, kind, span) // ops.DECODE_SPLIT + 1


def test_decode_split_bounds_hold_for_drawn_rows():
    r = random.Random(0)
    for _ in range(2000):
        kind = r.choice([ops.MASK_FULL, ops.MASK_CHUNK, ops.MASK_WINDOW])
        span = r.choice([1, 16, 100, 256, 257, 300, 512, 8192, 70000])
        rows = r.randint(1, 70)
        top = r.choice([1, 5, 255, 256, 257, 1000, 8192, 8193, 140000])
        positions = [r.randrange(top) for _ in range(rows)]
        max_context = max(positions) + 1
        per_row = ops.decode_splits(max_context, kind, span)
        need = [splits_of(p, kind, span) for p in positions]
        assert max(need) <= per_row, (kind, span, positions)
        # what attention_decode launches when it is told the rows' keys: never fewer CTAs than there are splits
        keys = sum(p + 1 for p in positions)
        items = min(rows * per_row, keys // ops.DECODE_SPLIT + rows)
        assert sum(need) <= items, (kind, span, positions)


def test_decode_split_bound_is_tight_for_whole_chunks():
    assert ops.decode_splits(8192, ops.MASK_FULL, 1) == 32
    assert ops.decode_splits(8193, ops.MASK_FULL, 1) == 33
    assert ops.decode_splits(1, ops.MASK_FULL, 1) == 1
    # a chunk of 8192 keys that starts on a split boundary never spans more than 33 splits, however long the row
    assert ops.decode_splits(10 ** 6, ops.MASK_CHUNK, 8192) == 33
    assert ops.decode_splits(100, ops.MASK_WINDOW, 700) == 1


def test_attention_planner_cuts_tiles_and_single_rows():
    """Portions become tiles of the planner's size, short entries single rows; the plan of a decode-only step
    has no arrays at all, so a replayed graph has nothing of it to refresh."""
    from sharpinference_b200.parts.attention import PagedAttentionPlanner
    p = PagedAttentionPlanner(64)
    d = p.plan([100, 7, 0, 33], [150, 1, 4, 5])
    assert d.arrays["tiles"].tolist() == [[0, 64, 100, 0], [64, 64, 164, 0], [128, 22, 228, 0], [155, 5, 33, 3]]
    assert d.arrays["decode_rows"].tolist() == [150, 151, 152, 153, 154]
    assert d.values == {"num_tiles": 4, "num_decode_rows": 5, "tile_rows": 64, "decode_keys": 8 + (1 + 2 + 3 + 4)}
    d = p.plan([10, 20, 30], [1, 1, 1], bucket=p.bucket([10, 20, 30], [1, 1, 1]))
    assert d.arrays["tiles"].shape == (0, 4) and d.arrays["decode_rows"].size == 0
    assert d.values["num_decode_rows"] == 3 and d.values["decode_keys"] == p.keys_bucket(63, 3) >= 63
    assert PagedAttentionPlanner(128).key != p.key


def test_keys_bucket_of_a_captured_decode_step():
    """A replayed graph's attention launch is sized by the bucket: never below the keys, at most an eighth (or
    256 keys a row) above; a batch that gains a key a row each step changes bucket every 256 steps at most."""
    from sharpinference_b200.parts.attention import PagedAttentionPlanner as StepRunner    # the bucket is the planner's
    for rows in (1, 3, 8, 64):
        for keys in list(range(rows, 3000, 7)) + [65080, 65536, 65537, 10 ** 6, 2 ** 31 - 5]:
            b = StepRunner.keys_bucket(keys, rows)
            assert b >= keys
            assert b - keys < max(512 * rows, keys // 8 + 1), (keys, rows)
            assert StepRunner.keys_bucket(b, rows) == b                       # a bucket is its own bucket
        start = 5 * rows
        buckets = [StepRunner.keys_bucket(start + rows * step, rows) for step in range(4096)]
        changes = sum(a != b for a, b in zip(buckets, buckets[1:]))
        assert changes <= 4096 // 256 + 1, (rows, changes)
    assert len({StepRunner.keys_bucket(8 * (8192 - 57 + i), 8) for i in range(58)}) == 1


def test_chunk_bounds_hold_for_drawn_steps():
    """Chunks of the requests of a step that run in chunks: the bound that sizes scratch and grids, from the step's totals alone,
    and no scratch where the longest request has too few rows."""
    r = random.Random(1)
    for _ in range(3000):
        kind, heads = r.choice(["mlstm", "ssd", "wkv"]), r.choice([1, 4, 8, 32, 64, 200])
        least = ops.chunked_least(kind, heads)
        assert least >= ops.CHUNKED_LEAST
        lens = [r.choice([1, 1, r.randint(1, 300), least - 1, least, least + 1, r.randint(1, 3000)]) for _ in range(r.randint(1, 12))]
        need = sum((n + 63) // 64 for n in lens if n >= least)
        for known in (None, max(lens)):
            got = ops._chunks(kind, sum(lens), len(lens), known, heads, 64, 64)
            assert got >= need, (kind, heads, lens)
            assert known is None or (got > 0) == (max(lens) >= least)


@pytest.mark.parametrize("channels,alone,shared", [(512, 1700, 1500), (1024, 1700, 1500), (2048, 1700, 1500), (4096, 1500, 1300),
                                                    (8192, 1286, 1000)])
def test_the_scans_border_follows_the_channels(channels, alone, shared):
    """A request that gains in chunks beside what a step of 2048 rows has left for another one, and one that loses there."""
    assert shared < ops.chunked_least("scan", channels) <= alone
    assert ops.chunked_least("scan", 1 << 16) == ops.chunked_least("scan", 8192) > ops.CHUNKED_LEAST


def test_what_is_walked_behind_the_chunks():
    """Whether a step with chunks leaves requests to walk, their rows and the longest one's: from the lengths, and without them safely."""
    r = random.Random(2)
    for _ in range(2000):
        kind, heads = r.choice(["mlstm", "ssd", "wkv", "scan"]), r.choice([1, 8, 64, 1000, 4096, 20000])
        least = ops.chunked_least(kind, heads)
        assert least >= ops.CHUNKED_LEAST
        lens = [r.choice([1, r.randint(1, 300), least - 1, least, least + 1]) for _ in range(r.randint(1, 8))]
        T = sum(lens) + r.choice([0, 0, 5])                   # rows may lie behind the last request's
        if max(lens) < least:
            continue                                          # no chunks
        rest = [n for n in lens if n < least]
        assert ops._chunk_border(kind, T, len(lens), max(lens), lens, heads) == (least, int(bool(rest)), sum(rest), max(rest, default=0))
        for known in (None, max(lens)):
            unknown = ops._chunk_border(kind, T, len(lens), known, None, heads)
            assert unknown[0] == least and unknown[1] >= int(bool(rest)) and unknown[2:] == (0, 0)
    for wrong in ([2000], [2000, 2000], [1, 1, 1]):
        with pytest.raises(ops.KernelError):
            ops._chunk_border("ssd", 3000, 2, 2000, wrong, 8)


def test_chunk_kernels_are_left_alone_beyond_their_sizes():
    """Steps and sizes that the walks take and the chunk kernels refuse are walked: more chunks than a grid's third extent, values whose
    memory has more than 2^24 elements a head, odd sizes and addresses."""
    assert ops._chunks("ssd", 1 << 22, 1, None, 8, 64, 64) == 0 and ops._chunks("ssd", 65535 * 64, 1, None, 8, 64, 64) == 65535
    assert ops._chunks("mlstm", 4096, 1, None, 1, 128, 1 << 17) > 0 and ops._chunks("mlstm", 4096, 1, None, 1, 128, (1 << 17) + 4) == 0
    assert ops._chunks("mlstm", 4096, 1, None, 8, 130, 64) == 0 and ops._chunks("mlstm", 4096, 1, None, 8, 128, 66) == 0
    assert ops._chunks("ssd", 4096, 1, None, 8, 64, 64, 4, 1) == 0


def test_small_products_are_an_engine_steps_own():
    """Inside of an engine's step, and in its thread alone, small products may run on the weight-streaming kernel; the model's
    weights carry no mark of it afterwards, also when the step failed."""
    import threading

    import pytest
    import torch
    from sharpinference_b200.parts.linear import Linear, engine_step
    lin = Linear(torch.zeros(16, 8, dtype=torch.bfloat16))
    seen = []
    with pytest.raises(ValueError):
        with engine_step(True):
            assert lin.small(1) and lin.small(16) and not lin.small(17)
            other = threading.Thread(target=lambda: seen.append(lin.small(1)))
            other.start()
            other.join()
            with engine_step(False):
                assert not lin.small(1)
            assert lin.small(1)
            raise ValueError
    assert seen == [False] and not lin.small(1) and not lin.stream_small
