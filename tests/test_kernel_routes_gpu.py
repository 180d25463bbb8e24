"""Calls that a rule on sizes sends to one kernel or another: both are the same numbers, at the borders of the rules."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from sharpinference_b200.kernels import ops as o
    return o


def rnd(*shape, seed=0, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed), dtype=torch.float32).to(DEV) * scale


# key sizes of every lane count (one not a multiple of 4 floats), value columns that leave a block's last ones empty, 1 and 3 rows
@pytest.mark.parametrize("heads,d,dv,rows", [(8, 128, 128, 1), (8, 126, 100, 3), (16, 64, 160, 1), (4, 30, 128, 1), (8, 128, 256, 8)])
def test_delta_walk_with_four_columns_is_the_walk_with_one(ops, heads, d, dv, rows):
    """From 1024 requests times heads on eight lanes hold four columns; the same requests in two halves hold one."""
    B = 1024 // heads + 3
    T, dp = B * rows, (d + 3) // 4 * 4
    qkv, beta, z = rnd(T, heads * (2 * d + dv), seed=1, scale=d ** -0.5), torch.sigmoid(rnd(T, heads, seed=2)), rnd(T, heads * d, seed=3)
    kw = dict(dt_bias=rnd(heads * d, seed=4), a_log=rnd(heads, seed=5), kv_heads=heads, heads=heads, d=d, dv=dv, max_rows=rows)
    first = torch.arange(B + 1, dtype=torch.int32, device=DEV) * rows
    slots = torch.arange(B - 1, -1, -1, dtype=torch.int32, device=DEV)
    state = rnd(B, heads, dv, dp, seed=6)
    state[..., d:] = 0.0
    state = state.view(B, -1).contiguous()
    other, got = state.clone(), None
    got = ops.delta_rule(qkv, beta, z, row_offsets=first, state_slots=slots, state=state, num_requests=B, **kw)
    half = B // 2
    for lo, hi in ((0, half), (half, B)):
        r = slice(lo * rows, hi * rows)
        one = ops.delta_rule(qkv[r].contiguous(), beta[r].contiguous(), z[r].contiguous(), row_offsets=first[: hi - lo + 1].contiguous(),
                             state_slots=slots[lo:hi].contiguous(), state=other, num_requests=hi - lo, **kw)
        assert torch.equal(got[r], one)
    assert torch.equal(state, other) and bool(torch.isfinite(got).all())


# states that fill a lane's pairs and that do not, channels behind the last block's, chunks with a short last one, walked requests between
@pytest.mark.parametrize("C,N,lens,raw", [(100, 16, [300, 1, 200, 64], True), (256, 10, [128, 191, 500], False), (130, 5, [1000], True),
                                          (4096, 16, [200, 2, 192], True), (64, 3, [7, 256], True)])
def test_selective_scan_in_chunks(ops, monkeypatch, C, N, lens, raw):
    """Outputs and state against the walk in 64 bits (the float32 walk itself is held to 2e-5 of the largest), a second portion from the
    first one's state, and every request's numbers those that it has alone."""
    monkeypatch.setitem(ops._WALK_OR_CHUNKS, "scan", (1e9, 1, 0.0))                            # in chunks from 128 rows on
    B, T = len(lens), sum(lens)
    x, z, bc = rnd(2 * T, C, seed=1), rnd(2 * T, C, seed=2), rnd(2 * T, 2 * N, seed=3)
    dt, bias = rnd(2 * T, C, seed=4), rnd(C, seed=5) - 3.0
    if not raw:
        dt = torch.nn.functional.softplus(dt - 3.0)
    a_log, dsk = torch.log(torch.arange(1, N + 1, dtype=torch.float32, device=DEV)).repeat(C, 1).contiguous(), rnd(C, seed=6)
    first = [sum(lens[:b]) for b in range(B + 1)]

    def run(rows, part, slots, state):
        off = torch.tensor([sum(part[:b]) for b in range(len(part) + 1)], dtype=torch.int32, device=DEV)
        return ops.selective_scan(x[rows], dt[rows], bc[rows], 0, N, a_log, dsk, z[rows], 0, row_offsets=off, state=state, split=True,
                                  state_slots=torch.tensor(slots, dtype=torch.int32, device=DEV), out_dtype=torch.float32,
                                  dt_bias=bias if raw else None, max_rows=max(part))
    state, alone, S = rnd(B, C * N, seed=7), rnd(B, C * N, seed=7), rnd(B, C * N, seed=7).double().view(B, C, N)
    for half in range(2):
        out = run(slice(half * T, half * T + T), lens, list(range(B)), state)
        for b in range(B):
            rows = slice(half * T + first[b], half * T + first[b + 1])
            one = run(rows, lens[b:b + 1], [b], alone)
            assert torch.equal(out[first[b]:first[b + 1]], one), b
            want = torch.empty(lens[b], C, dtype=torch.float64, device=DEV)
            d = dt[rows].double()
            d = torch.nn.functional.softplus(d + bias.double(), threshold=1e9) if raw else d
            g = z[rows].double()
            g = torch.nn.functional.silu(g) if raw else g
            xx, Bn, Cn = x[rows].double(), bc[rows, :N].double(), bc[rows, N:].double()
            for t in range(lens[b]):
                S[b] = torch.exp(-d[t][:, None] * a_log.double().exp()) * S[b] + (d[t] * xx[t])[:, None] * Bn[t]
                want[t] = (S[b] @ Cn[t] + dsk.double() * xx[t]) * g[t]
            assert float((one - want).abs().max()) < 2e-5 * float(want.abs().max()), b
        assert torch.equal(state, alone)
        assert float((state.view(B, C, N) - S).abs().max()) < 2e-5 * float(S.abs().max())
