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


# contexts of less, as many and more tiles of 64 keys than a cluster has CTAs, the last round without tiles for some; element groups of
# every width; a window with kept positions; keys-only pages
@pytest.mark.parametrize("d,planes,mask,span,keep", [(128, 2, 0, 1, 0), (64, 2, 1, 300, 0), (20, 1, 0, 1, 0), (256, 2, 2, 170, 70)])
def test_float32_attention_in_clusters_is_one_cta_a_row(ops, d, planes, mask, span, keep):
    """A few decode rows share their key tiles in clusters; the same rows in one launch with many more have a CTA each."""
    nq, nkv, ps, pages = 6, 2, 16, 70
    kv = rnd(pages, planes, nkv, ps, d, seed=d)
    table = torch.arange(pages, dtype=torch.int32, device=DEV).view(1, -1)
    some = [0, 63, 64, 130, 511, 512, 600, 1023, 1100]
    many = some + [t % 40 for t in range(600)]
    q = rnd(len(many), nq, d, seed=1)

    def run(n):
        pos = torch.tensor(many[:n], dtype=torch.int32, device=DEV)
        return ops.paged_attention_generic(q[:n].contiguous(), kv, table, torch.zeros_like(pos), pos, nq=nq, nkv=nkv, d=d, page_size=ps,
                                           mask_kind=mask, mask_span=span, scale=d ** -0.5, keep_first=keep)
    want = run(len(many))
    for n in (1, 3, len(some)):
        assert torch.equal(run(n), want[:n]), n


@pytest.mark.parametrize("sinks", [False, True])
def test_decode_rows_of_one_split_need_no_merge(ops, sinks):
    """bfloat16 decode rows of up to 256 keys: alone (they write their outputs themselves) and beside a longer row (a merge does)."""
    nq, nkv, d, ps = 8, 2, 128, 64
    kv = rnd(16, 2, nkv, ps, d, seed=1).bfloat16()
    table, pos = torch.arange(16, dtype=torch.int32, device=DEV).view(1, -1), torch.tensor([0, 255, 100, 700], dtype=torch.int32, device=DEV)
    q, sink = rnd(4, nq, d, seed=2).bfloat16(), rnd(nq, seed=3) * 4 if sinks else None
    keys, values = (kv[:, i].float().permute(1, 0, 2, 3).reshape(nkv, -1, d).double() for i in range(2))

    def run(n, context, most=None):
        out = torch.zeros(n, nq * d, dtype=torch.bfloat16, device=DEV)
        ops.attention_decode(q[:n].contiguous(), kv, table, torch.zeros(n, dtype=torch.int32, device=DEV), pos[:n].contiguous(), out, rows=None,
                             num_rows=n, nq=nq, nkv=nkv, d=d, page_size=ps, mask_kind=0, mask_span=1, scale=d ** -0.5,
                             max_context=context, max_keys=most, sinks=sink)
        return out
    full = run(4, 701)
    assert torch.equal(run(3, 256), full[:3]) and torch.equal(run(3, 1024, 358), full[:3]) and torch.equal(run(1, 1024, 256), full[:1])
    for r, p in enumerate(pos.tolist()):
        for h in range(nq):
            s = (keys[h // 4, : p + 1] @ q[r, h].double()) * d ** -0.5
            s = s if sink is None else torch.cat([s, sink[h: h + 1].double()])
            want = torch.softmax(s, dim=0)[: p + 1] @ values[h // 4, : p + 1]
            assert torch.allclose(full[r].view(nq, d)[h].double(), want, rtol=2e-2, atol=2e-2)


# (two million outputs: a denominator that is rounded otherwise moves about one bfloat16 in 60000)
@pytest.mark.parametrize("d,level", [(128, 6.0), (64, 2.0), (128, None)])
def test_decode_rows_of_one_split_are_the_bits_of_the_merge(ops, d, level):
    """Rows of up to 256 keys, most of them with sinks above their scores: alone, and in one launch with a longer row."""
    nq, nkv, ps, n = 8, 2, 64, 2000 * 128 // d
    kv, q = rnd(16, 2, nkv, ps, d, seed=1).bfloat16(), rnd(n + 1, nq, d, seed=2).bfloat16()
    table = torch.arange(16, dtype=torch.int32, device=DEV).view(1, -1)
    pos = torch.randint(0, 256, (n + 1,), generator=torch.Generator().manual_seed(3)).to(torch.int32).to(DEV)
    pos[n] = 700
    sink = None if level is None else rnd(nq, seed=4) + level

    def run(rows, context):
        out = torch.zeros(rows, nq * d, dtype=torch.bfloat16, device=DEV)
        ops.attention_decode(q[:rows].contiguous(), kv, table, torch.zeros(rows, dtype=torch.int32, device=DEV), pos[:rows].contiguous(), out,
                             rows=None, num_rows=rows, nq=nq, nkv=nkv, d=d, page_size=ps, mask_kind=0, mask_span=1, scale=d ** -0.5,
                             max_context=context, sinks=sink)
        return out
    assert torch.equal(run(n, 256), run(n + 1, 701)[:n])


# rows that fill a tile of activations and that do not, one and two weight tiles a CTA, output rows wider than the product, one head
@pytest.mark.parametrize("E,T,N,K,ld", [(3, 6, 40, 64, 48), (2, 130, 256, 128, 320), (8, 257, 300, 72, 300), (1, 33, 128, 256, 128)])
def test_product_a_head_with_the_heads_minor(ops, E, T, N, K, ld):
    """The bits of the float32 product turned and rounded; the columns behind the product stay as they are."""
    a, w = rnd(E * T, K, seed=1).bfloat16(), rnd(E, N, K, seed=2).bfloat16()
    out = torch.full((T, E, ld), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.tc_per_head(a, w, T, out)
    offsets = torch.arange(E + 1, dtype=torch.int32, device=DEV) * T
    want = ops.tc_grouped_gemm(a, w, offsets, mode=ops.TC_MODE_STORE).view(E, T, N).transpose(0, 1).to(torch.bfloat16)
    assert torch.equal(out[..., :N], want) and bool((out[..., N:] == 7.0).all())
    wide = torch.full((T, E, K + 16), float("nan"), dtype=torch.bfloat16, device=DEV)          # operand rows with the heads minor too
    wide[..., :K] = a.view(E, T, K).transpose(0, 1)
    again = torch.empty(T, E, N, dtype=torch.bfloat16, device=DEV)
    assert torch.equal(ops.tc_per_head(wide, w, T, again), want)


# every lane count, value columns behind the last block's and of several blocks, states behind the last lane's, several groups
@pytest.mark.parametrize("heads,groups,N,P", [(4, 1, 128, 64), (6, 3, 100, 36), (2, 2, 20, 100), (3, 1, 64, 4)])
def test_state_space_duality_step_is_the_walk(ops, heads, groups, N, P):
    """Rows that come one a step give the bits of the same rows in one portion, in the outputs and in the state."""
    B, rows, inner = 5, 3, heads * P
    xbc, dt = rnd(B * rows, inner + 2 * groups * N, seed=1), rnd(B * rows, heads, seed=2)
    kw = dict(col_x=0, col_b=inner, col_c=inner + groups * N, col_dt=0, dt_bias=rnd(heads, seed=3) - 2, a_log=rnd(heads, seed=4),
              dskip=rnd(heads, seed=5), heads=heads, groups=groups, states=N, vdim=P)
    slots = torch.tensor([3, 0, 4, 1, 2], dtype=torch.int32, device=DEV)
    whole = rnd(B, heads * N * P, seed=6)
    single = whole.clone()
    y = ops.ssd_scan(xbc, dt, row_offsets=torch.arange(B + 1, dtype=torch.int32, device=DEV) * rows, state_slots=slots, state=whole, **kw)
    for r in range(rows):
        at = torch.arange(B, device=DEV) * rows + r
        one = ops.ssd_scan(xbc[at].contiguous(), dt[at].contiguous(), row_offsets=torch.arange(B + 1, dtype=torch.int32, device=DEV),
                           state_slots=slots, state=single, **kw)
        assert torch.equal(one, y[at]), r
    assert torch.equal(single, whole)
    # as many rows as requests, dealt otherwise: one request has two, another none
    off = torch.tensor([0, 2, 2, 3, 4, 5], dtype=torch.int32, device=DEV)
    a, b = whole.clone(), whole.clone()
    got = ops.ssd_scan(xbc[:5], dt[:5], row_offsets=off, state_slots=slots, state=a, **kw)
    want = ops.ssd_scan(xbc[:2], dt[:2], row_offsets=off[:2].contiguous(), state_slots=slots[:1], state=b, **kw)
    assert torch.equal(got[:2], want) and torch.equal(a[3], b[3]) and torch.equal(a[0], whole[0])


@pytest.mark.parametrize("C,raw", [(256, True), (100, False), (33, True)])
def test_selective_scan_step_is_the_walk(ops, C, raw):
    """Rows that come one a step give the bits of the same rows in one portion, in the outputs and in the state."""
    B, rows, N = 7, 3, 16
    x, z, dt, bc = rnd(B * rows, C, seed=1), rnd(B * rows, C, seed=2), rnd(B * rows, C, seed=3), rnd(B * rows, 2 * N, seed=4)
    dt = dt if raw else torch.nn.functional.softplus(dt - 3.0)
    a_log, dsk, bias = rnd(C, N, seed=5), rnd(C, seed=6), rnd(C, seed=7) - 3.0
    slots = torch.tensor([3, 0, 6, 4, 1, 2, 5], dtype=torch.int32, device=DEV)

    def run(rows_of, off, sl, state):
        return ops.selective_scan(x[rows_of].contiguous(), dt[rows_of].contiguous(), bc[rows_of].contiguous(), 0, N, a_log, dsk,
                                  z[rows_of].contiguous(), 0, row_offsets=off, state_slots=sl, state=state, out_dtype=torch.float32,
                                  dt_bias=bias if raw else None)
    whole = rnd(B, C * N, seed=8)
    single, first = whole.clone(), torch.arange(B + 1, dtype=torch.int32, device=DEV)
    y = run(slice(0, B * rows), first * rows, slots, whole)
    for r in range(rows):
        at = torch.arange(B, device=DEV) * rows + r
        assert torch.equal(run(at, first, slots, single), y[at]), r
    assert torch.equal(single, whole)
    # as many rows as requests, dealt otherwise: one request has two, another none
    off = torch.tensor([0, 2, 2, 3, 4, 5, 6, 7], dtype=torch.int32, device=DEV)
    a, b = whole.clone(), whole.clone()
    got, want = run(slice(0, 7), off, slots, a), run(slice(0, 2), off[:2].contiguous(), slots[:1], b)
    assert torch.equal(got[:2], want) and torch.equal(a[3], b[3]) and torch.equal(a[0], whole[0])


@pytest.mark.parametrize("d,dv", [(128, 256), (40, 36), (132, 64), (256, 32)])
def test_matrix_memory_step_is_the_walk(ops, d, dv):
    """Rows that come one a step give the bits of the same rows in one portion, in the outputs and in the state."""
    B, rows, heads = 5, 3, 2
    ld = heads * (2 * d + dv) + 4
    proj, bias = rnd(B * rows, ld, seed=1), rnd(heads, seed=2)
    slots = torch.tensor([3, 0, 4, 1, 2], dtype=torch.int32, device=DEV)
    first = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    floats = ops.mlstm_state_floats(heads, d, dv)[1]

    def run(part, off, sl, state):
        return ops.mlstm_recurrence(part.contiguous(), col_q=0, col_k=heads * d, col_v=2 * heads * d, col_i=ld - 4, col_f=ld - 2,
                                    bias_i=bias, bias_f=bias + 1.0, row_offsets=off, state_slots=sl, state=state, heads=heads,
                                    d=d, dv=dv, cap=15.0, q_scale=d ** -0.5)
    whole = torch.zeros(B, floats, device=DEV)
    run(rnd(2 * B, ld, seed=3), first * 2, slots, whole)          # (a state that has seen rows)
    single, dealt = whole.clone(), whole.clone()
    want = run(proj, first * rows, slots, whole)
    for r in range(rows):
        at = torch.arange(B, device=DEV) * rows + r
        (num, nq, coef), (num_w, nq_w, coef_w) = run(proj[at], first, slots, single), want
        assert torch.equal(num, num_w[at]) and torch.equal(nq, nq_w[at]) and torch.equal(coef[..., :3], coef_w[at][..., :3]), r
    assert torch.equal(single, whole)
    # as many rows as requests, dealt otherwise: one request has two, another none
    off = torch.tensor([0, 2, 2, 3, 4, 5], dtype=torch.int32, device=DEV)
    before = dealt.clone()
    got = run(proj[:5], off, slots, dealt)
    alone = before.clone()
    want = run(proj[:2], off[:2].contiguous(), slots[:1].contiguous(), alone)
    assert torch.equal(got[0][:2], want[0]) and torch.equal(dealt[3], alone[3]) and torch.equal(dealt[0], before[0])


@pytest.mark.parametrize("split", [False, True])
def test_step_sizes_of_the_selective_scan(ops, split):
    """softplus of raw step sizes in [-30, 30], walked and in chunks, against 64 bits.  Rates so large that nothing is carried and ones
    elsewhere: an output is the step size times the gate, silu(64) = 64.  The bound is two units in the last place (2^-23 each at
    worst): what an exponential and a logarithm of float32 may be off, or the exponential and the roundings behind it in chunks."""
    T, C, N = 2048, 256, 16
    v = (torch.rand(T, C, generator=torch.Generator().manual_seed(1)) * 60 - 30).to(DEV)
    v[:1024] *= 0.25                                     # half of them in [-7.5, 7.5]
    v[0, 0] = 0.0
    bc = torch.zeros(T, 2 * N, device=DEV)
    bc[:, 0] = bc[:, N] = 1.0
    ones, off = torch.ones(T, C, device=DEV), torch.tensor([0, T], dtype=torch.int32, device=DEV)
    y = ops.selective_scan(ones, v, bc, 0, N, torch.full((C, N), 80.0, device=DEV), torch.zeros(C, device=DEV), 64.0 * ones, 0,
                           row_offsets=off, state_slots=off[:1], state=torch.zeros(1, C * N, device=DEV), out_dtype=torch.float32,
                           dt_bias=torch.zeros(C, device=DEV), max_rows=T, split=split)
    want = torch.clamp(v.double(), min=0) + torch.log1p(torch.exp(-v.double().abs()))
    assert float(((y.double() / 64 - want) / want).abs().max()) < 2 * 2.0 ** -23


def test_matrix_memory_gates_of_a_request_do_not_depend_on_its_company(ops):
    """A request of 60 rows: its gates are walked by a warp with helpers where it is alone, by one warp beside 100 single rows."""
    heads, d, dv, lens = 8, 32, 32, [60] + [1] * 100
    T, ld = sum(lens), 8 * 96 + 16
    proj, bias = rnd(T, ld, seed=1), rnd(heads, seed=2)
    floats = ops.mlstm_state_floats(heads, d, dv)[1]

    def run(n):
        rows, state = sum(lens[:n]), torch.zeros(n, floats, device=DEV)
        off = torch.tensor([sum(lens[:i]) for i in range(n + 1)], dtype=torch.int32, device=DEV)
        out = ops.mlstm_recurrence(proj[:rows].contiguous(), col_q=0, col_k=heads * d, col_v=2 * heads * d, col_i=ld - 16, col_f=ld - 8,
                                   bias_i=bias, bias_f=bias + 1.0, row_offsets=off, state_slots=torch.arange(n, dtype=torch.int32, device=DEV),
                                   state=state, heads=heads, d=d, dv=dv, cap=15.0, q_scale=d ** -0.5, max_rows=60)
        return (*out, state)
    alone, beside = run(1), run(len(lens))
    for a, b in zip(alone[:3], beside[:3]):
        n = 3 if a is alone[2] else None                     # (a row's and head's coefficients: the fourth place is empty)
        assert torch.equal(a[..., :n], b[:60, ..., :n])
    assert torch.equal(alone[3][0], beside[3][0])


# requests with a row less than the border between walk and chunks, that many and one more, beside single rows and short prompts
@pytest.mark.parametrize("kind", ["mlstm", "ssd", "wkv", "scan"])
@pytest.mark.parametrize("over", [[0, 0], [1, 0, None], [-1, 0], [-1, 1, None, None], [5, -1000]])
def test_recurrences_with_the_lengths_known(ops, monkeypatch, kind, over):
    """What the host knows of the requests' rows chooses kernels (none behind the chunks, the single rows' one, a walk) and no bit."""
    from sharpinference_b200.parts.mlstm import fused_mlstm_columns
    monkeypatch.setattr(ops, "_WALK_OR_CHUNKS", dict.fromkeys(ops._WALK_OR_CHUNKS, (1.0, 150, 0.0)))
    heads, d, dv, C, N = 2, 32, 32, 64, 16
    least = ops.chunked_least(kind, heads)
    lens = [1 if o is None else max(least + o, 3) for o in over]
    B, T, hd = len(lens), sum(lens), heads * d
    ins, vec = [rnd(T, hd, seed=i) for i in range(4)], [rnd(hd, scale=0.3, seed=9 + i) for i in range(3)]
    xbc, dt = rnd(T, heads * dv + 2 * d, scale=0.5, seed=7), rnd(T, C, seed=8)
    cols = fused_mlstm_columns(heads, d, dv)
    proj, bc, a_log = rnd(T, cols[-1], seed=6), rnd(T, 2 * N, seed=5), rnd(C, N, seed=4)
    floats = {"mlstm": ops.mlstm_state_floats(heads, d, dv)[1], "scan": C * N}.get(kind, heads * d * dv)

    def run(lengths):
        state = torch.zeros(B, floats, device=DEV)
        kw = dict(row_offsets=torch.tensor([sum(lens[:i]) for i in range(B + 1)], dtype=torch.int32, device=DEV), state=state,
                  state_slots=torch.arange(B, dtype=torch.int32, device=DEV), split=True, max_rows=max(lens), lengths=lengths)
        if kind == "scan":
            return ops.selective_scan(ins[0], dt, bc, 0, N, a_log, vec[0], ins[1], 0, out_dtype=torch.float32, dt_bias=vec[1], **kw), state
        kw["heads"] = heads
        if kind == "wkv":
            r, k, v, w = (x.clone() for x in ins)
            return ops.wkv_recurrence(r, k, v, w, vec[0], vec[1], d=d, **kw), state
        if kind == "ssd":
            return ops.ssd_scan(xbc, dt, col_x=0, col_b=heads * dv, col_c=heads * dv + d, col_dt=0, dt_bias=vec[0], a_log=vec[1],
                                dskip=vec[2], groups=1, states=d, vdim=dv, **kw), state
        return ops.mlstm_recurrence(proj, col_q=cols[0], col_k=cols[1], col_v=cols[2], col_i=cols[4], col_f=cols[5], bias_i=vec[0],
                                    bias_f=vec[1], d=d, dv=dv, cap=15.0, q_scale=d ** -0.5, **kw)[0], state
    assert max(lens) >= least
    for got, want in zip(run(lens), run(None)):
        assert torch.equal(got, want) and bool(torch.isfinite(got).all())
