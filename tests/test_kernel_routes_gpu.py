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
