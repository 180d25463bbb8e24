"""The work of this engine that is timed: whole sessions through ``Engine`` and single layers through the parts'
``forward``, over the sizes that the repository's own configurations and benchmark use.

A case is a dict of plain values.  ``kind`` names the path:

* ``session``: a small dense Llama 4 served end to end: prompts admitted, read in one step, then decoded a step at a time
  with given tokens (as replaying a trace does), the logits of every step returned.
* ``attention``: one grouped-query attention layer over the paged cache (projections, rotation, q/k norm, cache write,
  attention, output projection); ``rows`` new rows over ``requests`` requests that hold ``start`` positions each.
* ``moe``: one routed feed-forward, top-1 with a shared expert or top-k.
* ``mlstm``, ``wkv``, ``scan``, ``ssd``, ``delta``: one recurrent layer with its per-request state.
* ``latent``: one latent-attention layer from an empty cache.

In all layer cases ``rows`` rows are cut unevenly over ``requests`` requests; ``rows == requests`` is a decode step.
"""
import math
from types import SimpleNamespace

import torch

DEV = "cuda:0"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
PAGE = 64
EPS = 1e-5


# ---- the cases --------------------------------------------------------------------------------------------------
def listed():
    return [
        # One user of a small model: every step is a chain of short kernels and launches count.
        {"name": "session_one_user", "kind": "session", "dtype": "bfloat16", "width": 1024, "layers": 4, "requests": 1,
         "prompt": 100, "steps": 16},
        # The true 32-bit path (checking a model against another implementation): four users, ragged prompts.
        {"name": "session_float32", "kind": "session", "dtype": "float32", "width": 1024, "layers": 2, "requests": 4,
         "prompt": 301, "steps": 4},
        # A full batch decoding at long context with the flagship's layer sizes: the cache is streamed.
        {"name": "attention_decode", "kind": "attention", "width": 5120, "heads": 40, "kv_heads": 8, "requests": 64,
         "rows": 64, "start": 6000},
        # A portion of a long prompt at the same sizes: two thousand rows behind four thousand cached positions.
        {"name": "attention_prompt", "kind": "attention", "width": 5120, "heads": 40, "kv_heads": 8, "requests": 1,
         "rows": 2048, "start": 4096},
        # The mixture of the flagship over a prompt portion: sixteen experts of 8192 and the shared one.
        {"name": "moe_prompt", "kind": "moe", "width": 5120, "ff": 8192, "experts": 16, "top": 1, "rows": 2048},
        # A decode step of a top-2 mixture: nearly every expert's weights are streamed for a few rows each.
        {"name": "moe_decode", "kind": "moe", "width": 4096, "ff": 2048, "experts": 16, "top": 2, "rows": 24},
        # Prompts of three users in one step through the matrix memory.
        {"name": "mlstm_prompt", "kind": "mlstm", "width": 2048, "heads": 8, "requests": 3, "rows": 2051},
        # One long prompt through the WKV recurrence: nothing but its heads runs side by side.
        {"name": "wkv_prompt", "kind": "wkv", "width": 2048, "heads": 32, "requests": 1, "rows": 2048},
        # One long prompt through the selective scan.
        {"name": "scan_prompt", "kind": "scan", "width": 2048, "heads": 0, "requests": 1, "rows": 2048},
        # Two prompts through the state-space duality.
        {"name": "ssd_prompt", "kind": "ssd", "width": 2048, "heads": 64, "requests": 2, "rows": 1777},
        # One prompt through latent attention, read from an empty cache.
        {"name": "latent_prompt", "kind": "latent", "width": 2048, "heads": 16, "requests": 1, "rows": 2048},
        # Two hundred users decoding through the delta rule: the state is streamed.
        {"name": "delta_decode", "kind": "delta", "width": 2048, "heads": 16, "requests": 200, "rows": 200},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["session", "session", "attention", "attention", "moe", "moe", "mlstm", "wkv", "scan", "ssd",
                       "latent", "delta"])
    if kind == "session":
        if rng.random() < 0.5:
            return {"kind": kind, "dtype": "bfloat16", "width": rng.choice([512, 1024, 2048]), "layers": rng.randint(1, 5),
                    "requests": _log(rng, 1, 8), "prompt": _log(rng, 5, 400), "steps": rng.randint(4, 20)}
        return {"kind": kind, "dtype": "float32", "width": rng.choice([512, 1024]), "layers": rng.randint(1, 2),
                "requests": _log(rng, 1, 5), "prompt": _log(rng, 5, 400), "steps": rng.randint(1, 5)}
    if kind == "attention":
        width, heads = rng.choice([(5120, 40), (4096, 32), (2048, 16)])
        case = {"kind": kind, "width": width, "heads": heads, "kv_heads": heads // rng.choice([4, 5] if heads == 40 else [4, 8])}
        if rng.random() < 0.5:
            n = _log(rng, 8, 64)
            return dict(case, requests=n, rows=n, start=_log(rng, 500, 7900))
        return dict(case, requests=rng.randint(1, 4), rows=_log(rng, 200, 2048), start=rng.choice([0, _log(rng, 100, 5000)]))
    if kind == "moe":
        width, ff = rng.choice([(2048, 1024), (4096, 2048), (5120, 8192)])
        rows = _log(rng, 1, 64) if rng.random() < 0.5 else _log(rng, 200, 2048)
        return {"kind": kind, "width": width, "ff": ff, "experts": 16, "top": 1 if width == 5120 else rng.choice([1, 2]),
                "rows": rows}
    if kind == "latent":
        n = rng.randint(1, 3)
        return {"kind": kind, "width": 2048, "heads": rng.choice([8, 16]), "requests": n, "rows": _log(rng, 100, 2048)}
    width = rng.choice([1024, 2048])
    heads = {"mlstm": width // 256, "wkv": width // 64, "scan": 0, "ssd": width // 32, "delta": width // 128}[kind]
    if rng.random() < 0.35:
        n = _log(rng, 8, 200)
        return {"kind": kind, "width": width, "heads": heads, "requests": n, "rows": n}
    n = rng.randint(1, 4)
    return {"kind": kind, "width": width, "heads": heads, "requests": n, "rows": _log(rng, 150, 2048)}


# ---- sizes ------------------------------------------------------------------------------------------------------
def _cut(rows, requests):
    """``rows`` over ``requests`` requests, unevenly: shares of 1, 1/2, 1/3, ... and at least a row each."""
    if rows == requests:
        return [1] * rows
    share = [1.0 / (i + 1) for i in range(requests)]
    lengths = [max(1, int(rows * s / sum(share))) for s in share]
    lengths[0] += rows - sum(lengths)
    return lengths


def _starts(case):
    """Positions each request holds already: the decode batch of a server is at many places."""
    n = case["requests"]
    return [case["start"] - (i * 37) % max(1, case["start"] // 3) for i in range(n)]


def _prompts(case):
    """Lengths of a session's prompts."""
    return [max(1, case["prompt"] - (i * case["prompt"]) // (2 * case["requests"])) for i in range(case["requests"])]


class _Draws:
    """Seeded draws on the device; matrices as a checkpoint stores them."""

    def __init__(self, seed, dtype=BF16):
        self.g = torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + 17)
        self.dtype = dtype

    def matrix(self, *shape, std=0.02):
        return torch.empty(shape, dtype=self.dtype, device=DEV).normal_(0.0, std, generator=self.g)

    def vector(self, *shape, mean=0.0, std=0.1):
        return torch.empty(shape, dtype=F32, device=DEV).normal_(mean, std, generator=self.g)

    def acts(self, *shape):
        """Normed activations: unrounded, and as a product reads them."""
        x = torch.empty(shape, dtype=F32, device=DEV).normal_(0.0, 1.0, generator=self.g)
        return x, x.to(BF16)


# ---- weights and inputs, from the seed alone ----------------------------------------------------------------------
HEAD = 128                                   # head size of the attention layers, key size of mlstm and delta
LATENT = dict(dim=128, rot_dim=64, vdim=128, q_rank=768, kv_rank=256, rot_base=10000.0)
SCAN = dict(states=16, taps=4)
SSD = dict(vdim=64, states=128, groups=1, taps=4, norm_groups=1)


def _layer_tensors(case, seed):
    """The weights of a layer case and its input rows, by name."""
    r, kind, W = _Draws(seed), case["kind"], case["width"]
    t = {}
    t["h32"], t["h"] = r.acts(case["rows"], W)
    if kind == "attention":
        nq, nkv, d = case["heads"], case["kv_heads"], HEAD
        t["qkv"], t["o"] = r.matrix((nq + 2 * nkv) * d, W), r.matrix(W, nq * d)
    elif kind == "moe":
        E, ff = case["experts"], case["ff"]
        t["router"] = r.vector(E, W, std=0.02)
        t["gate_up"], t["down"] = r.matrix(E, 2 * ff, W), r.matrix(E, W, ff)
        t["shared_gate_up"], t["shared_down"] = r.matrix(2 * ff, W), r.matrix(W, ff)
    elif kind == "mlstm":
        heads, d, dv = case["heads"], HEAD, 2 * HEAD
        t["q"], t["k"], t["v"], t["g"] = r.matrix(heads * d, W), r.matrix(heads * d, W), r.matrix(heads * dv, W), r.matrix(heads * dv, W)
        t["i"], t["f"] = r.matrix(heads, W), r.matrix(heads, W)
        t["i.b"], t["f.b"] = r.vector(heads, mean=-1.0), r.vector(heads, mean=4.0, std=1.0)
        t["norm"], t["o"] = r.vector(heads * dv, mean=1.0), r.matrix(W, heads * dv)
    elif kind == "wkv":
        heads, d, rank = case["heads"], 64, 64
        t["mu"] = r.vector(5, W, mean=0.5, std=0.2)
        t["rkvg"] = r.matrix(4, heads * d, W)
        t["w1"], t["w2"] = r.matrix(rank, W), r.matrix(heads * d, rank, std=0.1)
        t["w0"], t["u"] = r.vector(heads * d, mean=-3.0, std=1.0), r.vector(heads * d)
        t["norm"], t["o"] = r.vector(heads * d, mean=1.0), r.matrix(W, heads * d)
    elif kind == "scan":
        inner, N, taps, rank = 2 * W, SCAN["states"], SCAN["taps"], W // 16
        t["in"], t["x"], t["dt"] = r.matrix(2 * inner, W), r.matrix(rank + 2 * N, inner), r.matrix(inner, rank, std=0.1)
        t["conv"], t["conv.b"] = r.vector(inner, taps, std=0.5), r.vector(inner)
        t["dt.b"], t["D"] = r.vector(inner, mean=-4.0, std=1.0), r.vector(inner, mean=1.0)
        t["A_log"] = torch.log(torch.arange(1, N + 1, dtype=F32, device=DEV)).repeat(inner, 1).contiguous()
        t["o"] = r.matrix(W, inner)
    elif kind == "ssd":
        heads, P, N, G, taps = case["heads"], SSD["vdim"], SSD["states"], SSD["groups"], SSD["taps"]
        inner, bc = heads * P, G * N
        t["in"] = r.matrix(2 * inner + 2 * bc + heads, W)
        t["conv"], t["conv.b"] = r.vector(inner + 2 * bc, taps, std=0.5), r.vector(inner + 2 * bc)
        t["dt.b"], t["A_log"], t["D"] = r.vector(heads, mean=-3.0, std=1.0), r.vector(heads, mean=1.0, std=0.7), r.vector(heads, mean=1.0)
        t["norm"], t["o"] = r.vector(inner, mean=1.0), r.matrix(W, inner)
    elif kind == "delta":
        heads, d, dv, taps, rank = case["heads"], HEAD, HEAD, 4, HEAD
        t["q"], t["k"], t["v"] = r.matrix(heads * d, W), r.matrix(heads * d, W), r.matrix(heads * dv, W)
        t["conv"] = r.vector(taps, heads * (2 * d + dv), std=0.5)
        t["a1"], t["g1"], t["b"] = r.matrix(rank, W), r.matrix(rank, W), r.matrix(heads, W)
        t["a2"], t["g2"] = r.matrix(heads * d, rank), r.matrix(heads * dv, rank)
        t["dt.b"], t["A_log"] = r.vector(heads * d, mean=-4.0, std=1.0), r.vector(heads, mean=0.5, std=0.5)
        t["norm"], t["o"] = r.vector(dv, mean=1.0), r.matrix(W, heads * dv)
    elif kind == "latent":
        H, d, dr, dv, rq, rk = case["heads"], LATENT["dim"], LATENT["rot_dim"], LATENT["vdim"], LATENT["q_rank"], LATENT["kv_rank"]
        t["dq"], t["dkv"], t["uq"] = r.matrix(rq, W), r.matrix(rk + dr, W), r.matrix(H * (d + dr), rq, std=0.04)
        t["dq.norm"], t["dkv.norm"] = r.vector(rq, mean=1.0), r.vector(rk, mean=1.0)
        t["uk"], t["uv"], t["o"] = r.matrix(H, d, rk, std=0.06), r.matrix(H, dv, rk, std=0.06), r.matrix(W, H * dv)
    return t


def _inv_freq(d, base):
    return base ** (-torch.arange(0, d, 2, dtype=F64) / d)


def _mixer(case, t):
    """The layer's mixer, put together from the framework's parts."""
    from sharpinference_b200 import parts as P
    kind, W = case["kind"], case["width"]
    if kind == "attention":
        rotary = P.RotaryEncoding(_inv_freq(HEAD, 500000.0).to(F32).to(DEV), "interleaved")
        return P.PagedAttention(qkv=P.Linear(t["qkv"]), out=P.Linear(t["o"]), num_heads=case["heads"],
                                num_kv_heads=case["kv_heads"], head_dim=HEAD, mask="chunk", span=8192, position=rotary,
                                qk_norm=P.L2Norm(EPS))
    if kind == "mlstm":
        heads, d, dv = case["heads"], HEAD, 2 * HEAD
        rows = [t["q"], t["k"], t["v"], t["g"], t["i"], t["f"]]
        pad = P.fused_mlstm_columns(heads, d, dv)[-1] - sum(x.shape[0] for x in rows)
        proj = torch.cat(rows + [torch.zeros((pad, W), dtype=BF16, device=DEV)])
        return P.MLSTMMixer(proj=P.Linear(proj), out=P.Linear(t["o"]), gate_bias_i=t["i.b"], gate_bias_f=t["f.b"],
                            head_norm_weight=t["norm"], heads=heads, key_dim=d, value_dim=dv, gate_cap=15.0, eps=EPS)
    if kind == "wkv":
        r, k, v, g = (P.Linear(x) for x in t["rkvg"])
        return P.WKVMixer(mu=t["mu"], r=r, k=k, v=v, g=g, w1=P.Linear(t["w1"]), w2=P.Linear(t["w2"]), w0=t["w0"], u=t["u"],
                          head_norm_weight=t["norm"], out=P.Linear(t["o"]), heads=case["heads"], head_dim=64, eps=EPS,
                          rkvg_weight=t["rkvg"])
    if kind == "scan":
        inner, N = 2 * W, SCAN["states"]
        return P.SelectiveScanMixer(in_proj=P.Linear(t["in"]), conv_weight=t["conv"], conv_bias=t["conv.b"],
                                    x_proj=P.Linear(t["x"]), dt_proj=P.Linear(t["dt"]), dt_bias=t["dt.b"], a_log=t["A_log"],
                                    d_skip=t["D"], out=P.Linear(t["o"]), inner=inner, states=N, dt_rank=W // 16, taps=SCAN["taps"])
    if kind == "ssd":
        return P.StateSpaceDualityMixer(in_proj=P.Linear(t["in"]), conv_weight=t["conv"], conv_bias=t["conv.b"],
                                        dt_bias=t["dt.b"], a_log=t["A_log"], d_skip=t["D"], norm_weight=t["norm"],
                                        out=P.Linear(t["o"]), heads=case["heads"], value_dim=SSD["vdim"], states=SSD["states"],
                                        groups=SSD["groups"], taps=SSD["taps"], norm_groups=SSD["norm_groups"], eps=EPS)
    if kind == "delta":
        heads, d, dv, low = case["heads"], HEAD, HEAD, 2 * HEAD
        rows = [t["q"], t["k"], t["v"], t["a1"], t["g1"], t["b"]]
        pad = P.delta_columns(heads, heads, d, dv, low)[-1] - sum(x.shape[0] for x in rows)
        proj = torch.cat(rows + [torch.zeros((pad, W), dtype=BF16, device=DEV)])
        up = torch.zeros((heads * (d + dv), low), dtype=BF16, device=DEV)
        up[: heads * d, : HEAD], up[heads * d:, HEAD:] = t["a2"], t["g2"]
        return P.ChannelDelta(proj=P.Linear(proj), up=P.Linear(up), out=P.Linear(t["o"]), conv_weight=t["conv"],
                              dt_bias=t["dt.b"], a_log=t["A_log"], norm_weight=t["norm"], heads=heads, kv_heads=heads, dim=d,
                              value_dim=dv, low=low, eps=EPS)
    m = LATENT
    rotary = P.RotaryEncoding(_inv_freq(m["rot_dim"], m["rot_base"]).to(F32).to(DEV), "interleaved", m["rot_dim"])
    return P.LatentAttention(down=P.Linear(torch.cat([t["dq"], t["dkv"]])), q_norm_weight=t["dq.norm"],
                             c_norm_weight=t["dkv.norm"], up_q=P.Linear(t["uq"]),
                             up_k=P.GroupedLinear(t["uk"].transpose(1, 2).contiguous()), up_v=P.GroupedLinear(t["uv"]),
                             out=P.Linear(t["o"]), num_heads=case["heads"], dim=m["dim"], rot_dim=m["rot_dim"],
                             value_dim=m["vdim"], q_rank=m["q_rank"], kv_rank=m["kv_rank"], eps=EPS,
                             softmax_scale=(m["dim"] + m["rot_dim"]) ** -0.5, position=rotary)


def _pages(starts, lengths):
    """Block tables as the cache manager deals pages out: the history of every request in turn, then the new rows."""
    tables, used = [], 0
    for s in starts:
        n = -(-s // PAGE)
        tables.append(list(range(used, used + n)))
        used += n
    for b, (s, n) in enumerate(zip(starts, lengths)):
        while len(tables[b]) < -(-(s + n) // PAGE):
            tables[b].append(used)
            used += 1
    return tables, used


def _history(case, seed, pages):
    """Keys and values that earlier steps left in the pages: keys of unit root mean square, as the q/k norm leaves them."""
    g = torch.Generator(device=DEV).manual_seed(7 * int(seed) + 3)
    return torch.empty((pages, 2, case["kv_heads"], PAGE, HEAD), dtype=BF16, device=DEV).normal_(0.0, 1.0, generator=g)


def _prepare_mixer(case, seed):
    from sharpinference_b200.cache import CacheManager
    from sharpinference_b200.engine.step import StepEntry, StepRunner
    from sharpinference_b200.models.model import ScheduleEntry
    t = _layer_tensors(case, seed)
    mixer = _mixer(case, t)
    lengths = _cut(case["rows"], case["requests"])
    starts = _starts(case) if case["kind"] == "attention" and case["start"] else [0] * len(lengths)
    _, pages = _pages(starts, lengths)
    blocks = [SimpleNamespace(mixer=mixer)]
    cache = CacheManager([ScheduleEntry(0)], blocks, page_size=PAGE, num_pages=pages, max_requests=len(lengths), dtype=BF16,
                         device=DEV)
    runner = StepRunner(SimpleNamespace(vocab_size=1 << 30, blocks=blocks), cache)
    for b in range(len(lengths)):
        cache.add_request(b)
    slot = cache.layer_slots()[0]
    if max(starts):
        slot.kv.copy_(_history(case, seed, pages))
        cache.reserve(list(enumerate(starts)))
        for b, s in enumerate(starts):
            cache.commit(b, s)
    cache.reserve(list(enumerate(lengths)))
    ctx = runner.build_context([StepEntry(b, [0] * n) for b, n in enumerate(lengths)])
    wide = mixer.wants_fp32_input
    return {"mixer": mixer, "ctx": ctx, "slot": slot, "h": t["h32"] if wide else t["h"], "cache": cache, "runner": runner}


def _run_mixer(s):
    slot = s["slot"]
    with torch.no_grad():
        y = s["mixer"].forward(s["ctx"], slot, s["h"])
    return {"y": y, "kv": slot.kv, "state": slot.state, "states": dict(slot.states)}


def _prepare_moe(case, seed):
    from sharpinference_b200 import parts as P
    t = _layer_tensors(case, seed)
    shared = P.DenseSwiGLU(gate_up=P.Linear(t["shared_gate_up"]), down=P.Linear(t["shared_down"]))
    kw = dict(router=t["router"], experts_gate_up=P.GroupedLinear(t["gate_up"]), experts_down=P.GroupedLinear(t["down"]), shared=shared)
    ffn = P.MoESigmoidTop1(act_dtype=BF16, **kw) if case["top"] == 1 else P.MoESigmoidTopKGated(top_k=case["top"], **kw)
    return {"ffn": ffn, "ctx": SimpleNamespace(extras={}, decode_only=case["rows"] <= 64), "h": t["h"], "h32": t["h32"]}


def _run_moe(s):
    with torch.no_grad():
        return s["ffn"].forward(s["ctx"], s["h"], s["h32"])


# ---- sessions ---------------------------------------------------------------------------------------------------
VOCAB = 8192


def _rope(layer):
    """Every fourth layer is global and does not rotate."""
    return (layer + 1) % 4 != 0


def _session_config(case):
    W, L = case["width"], case["layers"]
    return dict(architectures=["Llama4ForCausalLM"], vocab_size=VOCAB, hidden_size=W, num_hidden_layers=L,
                num_attention_heads=W // 128, num_key_value_heads=max(1, W // 512), head_dim=128, intermediate_size=4 * W,
                intermediate_size_mlp=4 * W, num_local_experts=1, num_experts_per_tok=1, moe_layers=[], rope_theta=500000.0,
                rope_scaling=None, no_rope_layers=[int(_rope(i)) for i in range(L)], attention_chunk_size=1024,
                use_qk_norm=True, attn_temperature_tuning=False, rms_norm_eps=EPS, tie_word_embeddings=True)


def _session_tensors(case, seed):
    """Every tensor of the model folder by name, and the tokens of the session."""
    c = _session_config(case)
    r = _Draws(seed, getattr(torch, case["dtype"]))
    H, d, nq, nkv, I = c["hidden_size"], 128, c["num_attention_heads"], c["num_key_value_heads"], c["intermediate_size_mlp"]
    w = {"model.embed_tokens.weight": r.matrix(VOCAB, H, std=0.05), "model.norm.weight": r.vector(H, mean=1.0)}
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, rows in (("q", nq * d), ("k", nkv * d), ("v", nkv * d)):
            w[f"{p}self_attn.{name}_proj.weight"] = r.matrix(rows, H, std=0.03)
        w[p + "self_attn.o_proj.weight"] = r.matrix(H, nq * d, std=0.03)
        for name, shape in (("gate", (I, H)), ("up", (I, H)), ("down", (H, I))):
            w[f"{p}feed_forward.{name}_proj.weight"] = r.matrix(*shape, std=0.03)
        for name in ("input_layernorm", "post_attention_layernorm"):
            w[f"{p}{name}.weight"] = r.vector(H, mean=1.0)
    g = torch.Generator().manual_seed(int(seed) + 5)
    prompts = [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in _prompts(case)]
    follow = torch.randint(0, VOCAB, (case["steps"], case["requests"]), generator=g).tolist()
    return c, w, prompts, follow


def _session_source(tensors, dtype):
    """The framework's weight interface over tensors at hand: what a program brings that keeps weights of its own."""
    from sharpinference_b200.weights.source import WeightSource

    class AtHand(WeightSource):
        compute_dtype, device = dtype, torch.device(DEV)

        def matrix(self, name, shape):
            return tensors[name].to(dtype)

        def vector(self, name, shape, init="norm"):
            return tensors[name].to(F32)

        def stored(self, name):
            return name in tensors

    return AtHand()


def _prepare_session(case, seed):
    from sharpinference_b200 import Engine, EngineOptions, StepEntry, get_architecture
    c, w, prompts, follow = _session_tensors(case, seed)
    arch = get_architecture("Llama4ForCausalLM")
    dtype = getattr(torch, case["dtype"])
    model = arch.build(arch.config_cls.from_dict(c), _session_source(w, dtype))
    tokens = sum(len(p) + case["steps"] for p in prompts)
    engine = Engine(model, dtype=case["dtype"], device=DEV,
                    options=EngineOptions(page_size=PAGE, max_cache_tokens=tokens + 2 * PAGE * len(prompts),
                                          max_batch=len(prompts), max_tokens_per_step=sum(map(len, prompts))))
    state = {"engine": engine, "prompts": [[(t * 7 + 1) % VOCAB for t in p] for p in prompts], "follow": follow, "entry": StepEntry}
    _run_session(state)                       # a server that has been up: its decode steps are captured
    return dict(state, prompts=prompts)


def _run_session(s):
    engine, entry, prompts = s["engine"], s["entry"], s["prompts"]
    for b in range(len(prompts)):
        engine.open_request(b)
    logits = [engine.forward_step([entry(b, p, [len(p) - 1]) for b, p in enumerate(prompts)])]
    for step in s["follow"]:
        # a replayed step leaves its logits in a buffer of its own, which the next one overwrites
        logits.append(engine.forward_step([entry(b, [t], [0]) for b, t in enumerate(step)]).clone())
    for b in range(len(prompts)):
        engine.close_request(b)
    return torch.stack(logits)


def prepare(case, seed):
    if case["kind"] == "session":
        return dict(_prepare_session(case, seed), run=_run_session)
    if case["kind"] == "moe":
        return dict(_prepare_moe(case, seed), run=_run_moe)
    return dict(_prepare_mixer(case, seed), run=_run_mixer)


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def work(case):
    kind, W = case["kind"], case["width"]
    if kind == "session":
        size = 2 if case["dtype"] == "bfloat16" else 4
        d, nkv, I, L = 128, max(1, W // 512), 4 * W, case["layers"]
        weights = L * ((2 * W + 2 * nkv * d) * W + 3 * W * I) + VOCAB * W
        prompts, B, n = _prompts(case), case["requests"], case["steps"]
        cached = sum(sum(min(p + i + 1, 1024) for i in range(n)) for p in prompts) * 2 * nkv * d * L * size
        rows = sum(prompts) + B * n
        pairs = sum(p * (p + 1) / 2 for p in prompts) + sum(p * n + n * (n + 1) / 2 for p in prompts)
        flops = 2 * rows * (weights - VOCAB * W) + 2 * B * (n + 1) * VOCAB * W + 4 * W * pairs * L
        return {"bytes": (n + 1) * weights * size + cached + rows * W * size + B * (n + 1) * VOCAB * 4, "flops": flops}
    T = case["rows"]
    io = T * W * (2 + 4)                         # the normed rows in, the float32 output out
    if kind == "moe":
        E, ff, top = case["experts"], case["ff"], case["top"]
        used = E * (1 - (1 - top / E) ** T)      # experts that the rows touch, uniformly routed
        return {"bytes": (used + 1) * 3 * W * ff * 2 + E * W * 4 + io + T * W * 4,
                "flops": 2 * T * (top + 1) * 3 * W * ff + 2 * T * E * W}
    lengths = _cut(T, case["requests"])
    if kind == "attention":
        nq, nkv = case["heads"], case["kv_heads"]
        starts = _starts(case) if case["start"] else [0] * len(lengths)
        pairs = sum(n * s + n * (n + 1) / 2 for s, n in zip(starts, lengths))
        weights = (2 * nq + 2 * nkv) * HEAD * W
        return {"bytes": weights * 2 + io + sum(s + 2 * n for s, n in zip(starts, lengths)) * 2 * nkv * HEAD * 2,
                "flops": 2 * T * weights + 4 * nq * HEAD * pairs}
    if kind == "latent":
        H, d, dr, dv, rq, rk = case["heads"], LATENT["dim"], LATENT["rot_dim"], LATENT["vdim"], LATENT["q_rank"], LATENT["kv_rank"]
        weights = (rq + rk + dr) * W + H * (d + dr) * rq + H * (d + dv) * rk + W * H * dv
        pairs = sum(n * (n + 1) / 2 for n in lengths)
        # scores and sums in the heads' own sizes; the keys and values of a row are expanded once
        return {"bytes": weights * 2 + io + 2 * T * (rk + dr) * 2, "flops": 2 * T * weights + 2 * H * (d + dr + dv) * pairs}
    heads = case["heads"]
    if kind == "mlstm":
        d, dv = HEAD, 2 * HEAD
        weights, state, per_row = heads * (2 * d + 2 * dv + 2) * W + W * heads * dv, heads * (d * dv + d + 1), 4 * heads * d * (dv + 1)
    elif kind == "wkv":
        d = 64
        weights, state, per_row = 5 * heads * d * W + 64 * (W + heads * d), heads * d * d + W, 4 * heads * d * d
    elif kind == "scan":
        inner, N, rank = 2 * W, SCAN["states"], W // 16
        weights = 3 * inner * W + (2 * rank + 2 * N) * inner
        state, per_row = inner * (N + SCAN["taps"] - 1), 6 * inner * N + 2 * inner * SCAN["taps"]
    elif kind == "ssd":
        P, N, G = SSD["vdim"], SSD["states"], SSD["groups"]
        inner, ch = heads * P, heads * P + 2 * G * N
        weights = (inner + ch + heads + inner) * W
        state, per_row = heads * N * P + (SSD["taps"] - 1) * ch, 4 * inner * N + 2 * ch * SSD["taps"]
    else:                                       # delta
        d, dv = HEAD, HEAD
        ch = heads * (2 * d + dv)
        weights = (ch + 2 * HEAD + heads) * W + heads * (d + dv) * HEAD + W * heads * dv
        state, per_row = heads * d * dv + 3 * ch, 7 * heads * d * dv + 2 * ch * 4
    return {"bytes": weights * 2 + io + 2 * len(lengths) * state * 4, "flops": 2 * T * weights + T * per_row}


def tolerance(case):
    # Four times the error seen against ``exact`` on B200, over listed and drawn cases: bfloat16 rounding of activations
    # and of what enters a product.  A whole model of a few layers in bfloat16: 1.1e-2.  Layers: 1.7e-3, and 2.6e-3 to
    # 4.2e-3 where probabilities, latents or shifted inputs are rounded on the way.  The 32-bit session: 3.5e-6.
    if case["kind"] == "session":
        return {"rel": 0.03} if case["dtype"] == "bfloat16" else {"rel": 1.4e-5}
    return {"rel": 0.016} if case["kind"] in ("attention", "latent", "wkv") else {"rel": 0.007}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _rotate(x, positions, base):
    """Neighbouring pairs of the last axis of ``x [T, heads, d]`` turned by position times frequency."""
    ang = positions.to(F64)[:, None, None] * _inv_freq(x.shape[-1], base).to(x.device)
    c, s, a, b = torch.cos(ang), torch.sin(ang), x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)


def _attend(q, k, v, first, scale):
    """``q [n, H, d]`` at positions ``first ..`` over ``k, v [S, G, *]``: grouped heads, causal."""
    n, H = q.shape[:2]
    rep = H // k.shape[1]
    out = torch.empty((n, H, v.shape[-1]), dtype=F64, device=q.device)
    see = torch.arange(k.shape[0], device=q.device)[None, :] <= first + torch.arange(n, device=q.device)[:, None]
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].T) * scale
        out[:, h] = torch.softmax(s.masked_fill(~see, -math.inf), dim=-1) @ v[:, h // rep]
    return out


def _conv(x, w, b=None):
    """Causal convolution per channel (``w [channels, taps]``, the last column the current row's), zeros before the start."""
    taps = w.shape[1]
    xp = torch.cat([torch.zeros((taps - 1, x.shape[1]), dtype=F64, device=x.device), x])
    y = sum(xp[j: j + x.shape[0]] * w[:, j] for j in range(taps))
    return y if b is None else y + b


def _exact_attention(case, seed, t, lengths):
    nq, nkv, d = case["heads"], case["kv_heads"], HEAD
    starts = _starts(case) if case["start"] else [0] * len(lengths)
    tables, pages = _pages(starts, lengths)
    old = _history(case, seed, pages) if max(starts) else None
    x = t["h"] @ t["qkv"].T
    out, r = [], 0
    for b, (s, n) in enumerate(zip(starts, lengths)):
        pos = torch.arange(s, s + n, device=DEV)
        q, k, v = x[r: r + n].split([nq * d, nkv * d, nkv * d], dim=1)
        q, k = (_rms(_rotate(z.reshape(n, -1, d), pos, 500000.0)) for z in (q, k))
        v = v.reshape(n, nkv, d)
        if s:
            past = old[torch.tensor(tables[b], device=DEV)].to(F64).permute(1, 0, 3, 2, 4).reshape(2, -1, nkv, d)[:, :s]
            k, v = torch.cat([past[0], k]), torch.cat([past[1], v])
        out.append(_attend(q, k, v, s, d ** -0.5).reshape(n, nq * d))
        r += n
    return torch.cat(out) @ t["o"].T


def _exact_moe(case, t):
    h, ff = t["h"], case["ff"]
    score = torch.sigmoid(t["h32"] @ t["router"].T)
    w, chosen = torch.topk(score, case["top"], dim=1)

    def net(x, gate_up, down):
        gu = x @ gate_up.to(F64).T
        return (_silu(gu[:, :ff]) * gu[:, ff:]) @ down.to(F64).T
    y = net(h, t["shared_gate_up"], t["shared_down"])
    for e in range(case["experts"]):
        rows, which = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            y[rows] += net(h[rows] * w[rows, which][:, None], t["gate_up"][e], t["down"][e])
    return y


def _exact_mlstm(case, t, h):
    T, H, d, dv = h.shape[0], case["heads"], HEAD, 2 * HEAD
    q, k = (h @ t["q"].T).view(T, H, d) * d ** -0.5, (h @ t["k"].T).view(T, H, d)
    v = (h @ t["v"].T).view(T, H, dv)
    i = 15.0 * torch.tanh((h @ t["i"].T + t["i.b"]) / 15.0)
    f = torch.nn.functional.logsigmoid(15.0 * torch.tanh((h @ t["f"].T + t["f.b"]) / 15.0))
    S, n, m = (torch.zeros(s, dtype=F64, device=DEV) for s in ((H, d, dv), (H, d), (H,)))
    o = torch.empty((T, H, dv), dtype=F64, device=DEV)
    for r in range(T):
        new = torch.maximum(f[r] + m, i[r])
        keep, take = torch.exp(f[r] + m - new), torch.exp(i[r] - new)
        S = keep[:, None, None] * S + (take[:, None] * k[r])[:, :, None] * v[r][:, None, :]
        n, m = keep[:, None] * n + take[:, None] * k[r], new
        den = torch.maximum((n * q[r]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        o[r] = (S * q[r][:, :, None]).sum(1) / den[:, None]
    return (_rms(o).reshape(T, -1) * t["norm"] * torch.sigmoid(h @ t["g"].T)) @ t["o"].T


def _exact_wkv(case, t, h):
    T, H, d = h.shape[0], case["heads"], 64
    prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    r, k, v, g, wm = (h + (prev - h) * t["mu"][s] for s in range(5))
    r, k, v = ((x @ t["rkvg"][s].T).view(T, H, d) for s, x in enumerate((r, k, v)))
    gate = _silu(g @ t["rkvg"][3].T)
    w = torch.exp(-torch.exp(torch.tanh(wm @ t["w1"].T) @ t["w2"].T + t["w0"])).view(T, H, d)
    u = t["u"].view(H, d)
    S, o = torch.zeros((H, d, d), dtype=F64, device=DEV), torch.empty((T, H, d), dtype=F64, device=DEV)
    for i in range(T):
        kv = k[i][:, :, None] * v[i][:, None, :]
        o[i] = ((S + u[:, :, None] * kv) * r[i][:, :, None]).sum(1)
        S = w[i][:, :, None] * S + kv
    return (_rms(o).reshape(T, -1) * t["norm"] * gate) @ t["o"].T


def _exact_scan(case, t, h):
    T, inner, N, rank = h.shape[0], 2 * case["width"], SCAN["states"], case["width"] // 16
    xz = h @ t["in"].T
    x, z = _silu(_conv(xz[:, :inner], t["conv"], t["conv.b"])), xz[:, inner:]
    dt, B, C = (x @ t["x"].T).split([rank, N, N], dim=1)
    dt = torch.nn.functional.softplus(dt @ t["dt"].T + t["dt.b"], threshold=1e9)
    A = -torch.exp(t["A_log"])
    S, y = torch.zeros((inner, N), dtype=F64, device=DEV), torch.empty((T, inner), dtype=F64, device=DEV)
    for i in range(T):
        S = torch.exp(dt[i][:, None] * A) * S + (dt[i] * x[i])[:, None] * B[i]
        y[i] = S @ C[i] + t["D"] * x[i]
    return (y * _silu(z)) @ t["o"].T


def _exact_ssd(case, t, h):
    T, H, P, N = h.shape[0], case["heads"], SSD["vdim"], SSD["states"]
    inner = H * P
    xbc, z, dt = (h @ t["in"].T).split([inner + 2 * N, inner, H], dim=1)
    x, B, C = _silu(_conv(xbc, t["conv"], t["conv.b"])).split([inner, N, N], dim=1)
    x, dt = x.reshape(T, H, P), torch.nn.functional.softplus(dt + t["dt.b"], threshold=1e9)
    decay = torch.exp(-torch.exp(t["A_log"]) * dt)
    S, y = torch.zeros((H, N, P), dtype=F64, device=DEV), torch.empty((T, H, P), dtype=F64, device=DEV)
    for i in range(T):
        S = decay[i][:, None, None] * S + dt[i][:, None, None] * B[i][None, :, None] * x[i][:, None, :]
        y[i] = (S * C[i][None, :, None]).sum(1) + t["D"][:, None] * x[i]
    return (_rms(y.reshape(T, inner) * _silu(z)) * t["norm"]) @ t["o"].T


def _exact_delta(case, t, h):
    T, H, d, dv = h.shape[0], case["heads"], HEAD, HEAD
    w = t["conv"].T
    q, k, v = (_silu(_conv(h @ t[s].T, w[i * H * d: (i + 1) * H * d])).view(T, H, d) for i, s in enumerate("qkv"))
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q = q * d ** -0.5
    b = torch.sigmoid(h @ t["b"].T)
    step = torch.nn.functional.softplus((h @ t["a1"].T) @ t["a2"].T + t["dt.b"], threshold=1e9).view(T, H, d)
    g = torch.exp(-torch.exp(t["A_log"])[None, :, None] * step)
    gate = torch.sigmoid((h @ t["g1"].T) @ t["g2"].T)
    S, o = torch.zeros((H, d, dv), dtype=F64, device=DEV), torch.empty((T, H, dv), dtype=F64, device=DEV)
    for i in range(T):
        S = g[i][:, :, None] * S
        u = b[i][:, None] * (v[i] - (S * k[i][:, :, None]).sum(1))
        S = S + k[i][:, :, None] * u[:, None, :]
        o[i] = (S * q[i][:, :, None]).sum(1)
    return ((_rms(o) * t["norm"]).reshape(T, -1) * gate) @ t["o"].T


def _exact_latent(case, t, h):
    T, H, d, dr, dv, rk, base = (h.shape[0], case["heads"], LATENT["dim"], LATENT["rot_dim"], LATENT["vdim"], LATENT["kv_rank"],
                                 LATENT["rot_base"])
    pos = torch.arange(T, device=DEV)
    q = ((_rms(h @ t["dq"].T) * t["dq.norm"]) @ t["uq"].T).view(T, H, d + dr)
    c, kr = (h @ t["dkv"].T).split([rk, dr], dim=1)
    c = _rms(c) * t["dkv.norm"]
    k = torch.cat([torch.einsum("tr,hdr->thd", c, t["uk"]), _rotate(kr[:, None], pos, base).expand(T, H, dr)], dim=-1)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], pos, base)], dim=-1)
    o = _attend(q, k, torch.einsum("tr,hvr->thv", c, t["uv"]), 0, (d + dr) ** -0.5)
    return o.reshape(T, H * dv) @ t["o"].T


def _exact_session(case, seed):
    c, w, prompts, follow = _session_tensors(case, seed)
    w = {k: v.to(F64) for k, v in w.items()}
    nq, nkv, d = c["num_attention_heads"], c["num_key_value_heads"], 128
    out = []
    for b, prompt in enumerate(prompts):
        toks = torch.tensor(prompt + [step[b] for step in follow], device=DEV)
        x, n = w["model.embed_tokens.weight"][toks], toks.numel()
        pos = torch.arange(n, device=DEV)
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = _rms(x) * w[p + "input_layernorm.weight"]
            q, k, v = ((h @ w[f"{p}self_attn.{s}_proj.weight"].T).view(n, -1, d) for s in "qkv")
            if _rope(i):
                q, k = (_rms(_rotate(z, pos, 500000.0)) for z in (q, k))
            x = x + _attend(q, k, v, 0, d ** -0.5).reshape(n, nq * d) @ w[p + "self_attn.o_proj.weight"].T
            h = _rms(x) * w[p + "post_attention_layernorm.weight"]
            gate, up, down = (w[f"{p}feed_forward.{s}_proj.weight"] for s in ("gate", "up", "down"))
            x = x + (_silu(h @ gate.T) * (h @ up.T)) @ down.T
        out.append((_rms(x[len(prompt) - 1:]) * w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T)
    return torch.stack(out, dim=1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "session":
        return _exact_session(case, seed)
    t = _layer_tensors(case, seed)
    if kind == "moe":
        t.update({k: t[k].to(F64) for k in ("h", "h32", "router")})          # the experts one at a time
        return _exact_moe(case, t)
    if kind == "wkv":
        t["h"] = t["h32"]
    t = {k: v.to(F64) for k, v in t.items()}
    lengths = _cut(case["rows"], case["requests"])
    if kind == "attention":
        return {"y": _exact_attention(case, seed, t, lengths), "kv": None, "state": None, "states": None}
    one = {"mlstm": _exact_mlstm, "wkv": _exact_wkv, "scan": _exact_scan, "ssd": _exact_ssd, "delta": _exact_delta,
           "latent": _exact_latent}[kind]
    y = torch.cat([one(case, t, t["h"][a: a + n]) for a, n in zip([sum(lengths[:i]) for i in range(len(lengths))], lengths)])
    return {"y": y, "kv": None, "state": None, "states": None}
