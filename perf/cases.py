"""The work this framework is given, as cases that can be timed and checked.

A case is one sublayer stack of a served model between its dense projections, on one step of the continuous-batching loop: some
entries decode one token each, others bring a portion of their prompt.  Four kinds:

    int8     quantize-on-write and attention over the paged int8 cache (HostDecodeStep for pure decode, scaffold.attention_ops
             for steps with prompt portions), `layers` layers on one step's metadata
    paged    Radivik's rotation, cache write and attention over the paged unquantised cache, bf16 or fp32
    experts  Radivik's feed-forward half: embedding, residual and norm, routed mixture of experts, residual and norm
    state    Biranex's mixers: windowed attention beside a state-space layer (`parallel`), the gated delta rule (`delta`)

Steps are recorded once into a CUDA graph and replayed, as the engine does for every bucket; `graph` False runs the calls one by
one, as the engine does for a step that fits no bucket.  `chained`: kernels may be brought up ahead of their predecessors' end
(kernels.set_early_start).  Entry lengths come from the case alone, everything else from the seed.
"""
from __future__ import annotations

import math
import random

import torch

from inference_engine_b200 import kernels as K
from inference_engine_b200 import ops
from inference_engine_b200 import scaffold as S
from inference_engine_b200.host_step import HostDecodeStep

EPS = 1e-6
GATE_SLOPE = 1.702
WIDTH = 2048
VOCAB = 32768
PAGE = 64  # page size of the unquantised caches

# "A" are the sizes of the int8 decoder, "B" smaller heads, more experts, one group of state channels
PAGED = {"A": (16, 8, 128, 128, 128), "B": (16, 8, 112, 96, 32)}  # heads, kv heads, key size, value size, rotated channels
EXPERTS = {"A": (8, 2, 3072), "B": (32, 4, 1536)}  # experts, chosen per token, feed-forward size
PARALLEL = {"A": (16, 8, 128, 128, 1024, 128, 64, 8, 128, 64), "B": (32, 8, 64, 64, 512, 32, 48, 1, 64, 64)}
# ^ attention heads, kv heads, key size, value size, window, rotated channels; state heads, groups, state channels, value size
DELTA = {"A": (16, 16, 128, 128), "B": (12, 6, 96, 112)}  # heads, key heads, key size, value size
TAPS = 4


# ----------------------------------------------------------------------------- the cases
def _case(kind, name=None, *, decoders=0, ctx_lo=0, ctx_hi=0, portions=0, rows=0, prior=0, graph=True, chained=False, **more):
    c = {"kind": kind, "decoders": decoders, "ctx_lo": ctx_lo, "ctx_hi": ctx_hi, "portions": portions, "rows": rows, "prior": prior,
         "graph": graph, "chained": chained, **more}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # a single chat turn decoding over a short history: launches and latency
        _case("int8", "int8_decode_1x300", decoders=1, ctx_lo=300, ctx_hi=300, layers=4, page=16, chained=True),
        # the reference's headline cell: a full batch of equal contexts
        _case("int8", "int8_decode_64x4096", decoders=64, ctx_lo=4096, ctx_hi=4096, layers=2, page=16, chained=True),
        # a batch as traffic leaves it: an odd count, contexts spread over two orders of magnitude
        _case("int8", "int8_decode_ragged_37", decoders=37, ctx_lo=90, ctx_hi=9000, layers=3, page=16),
        # the reference engine's mixed step: decoders beside one long portion of a prompt that is partly cached
        _case("int8", "int8_mixed_1024", decoders=32, ctx_lo=128, ctx_hi=4096, portions=1, rows=992, prior=3072, layers=1, page=16),
        # several new prompts of odd lengths at once: first portions, whose key calibration is made from them
        _case("int8", "int8_prompts_5", portions=5, rows=1011, layers=2, page=16),
        # the same mixed step over the unquantised cache
        _case("paged", "paged_mixed_1024", decoders=32, ctx_lo=1024, ctx_hi=4096, portions=1, rows=992, prior=3072, sizes="A", dtype="bf16"),
        # a prompt in full precision, as recorded traces are replayed: call by call
        _case("paged", "paged_fp32_prompt_200", portions=1, rows=200, prior=0, sizes="B", dtype="fp32", graph=False),
        # the feed-forward of a decode batch: the weights of every expert are streamed
        _case("experts", "experts_decode_64", decoders=64, ctx_lo=1, ctx_hi=1, sizes="A", dtype="bf16"),
        # and of a prompt step over many small experts
        _case("experts", "experts_prompt_1024", portions=1, rows=1024, sizes="B", dtype="bf16"),
        # a prompt portion through windowed attention and the state-space layer
        _case("state", "parallel_prompt_1024", portions=1, rows=1024, prior=1500, sizes="A", parallel=True, delta=False),
        # new prompts of odd lengths through the delta rule
        _case("state", "delta_prompts_3", portions=3, rows=1000, sizes="A", parallel=False, delta=True),
        # a decode batch through one layer of each kind
        _case("state", "state_decode_64", decoders=64, ctx_lo=200, ctx_hi=4096, sizes="B", parallel=True, delta=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: batches of 1 to 64 decoding entries of 32 to 4096 tokens, prompt steps of up to 1024 rows."""
    kind = rng.choice(["int8", "int8", "paged", "experts", "state"])
    shape = rng.choice(["decode", "decode", "prompt", "mixed"])
    step = {"graph": rng.random() < 0.85, "chained": rng.random() < 0.4}
    if shape != "prompt":
        lo, hi = sorted(_log(rng, 32, 4096) for _ in range(2))
        step.update(decoders=_log(rng, 1, 64 if shape == "decode" else 32), ctx_lo=lo, ctx_hi=hi)
    if shape != "decode":
        n = rng.randint(1, 5)
        step.update(portions=n, rows=_log(rng, 16 * n, 1000), prior=rng.choice([0, _log(rng, 40, 3072)]))
    if kind == "int8":
        return _case(kind, layers=rng.randint(1, 2), page=rng.choice([16, 16, 64]), **step)
    sizes, dtype = rng.choice("AB"), "bf16"
    if kind == "paged" and rng.random() < 0.25:  # full precision serves traces, not traffic: small steps
        dtype = "fp32"
        step.update(decoders=min(step.get("decoders", 0), 8), ctx_lo=min(step.get("ctx_lo", 0), 512), ctx_hi=min(step.get("ctx_hi", 0), 600),
                    rows=min(step.get("rows", 0), 200), prior=min(step.get("prior", 0), 300))
    if kind == "state":
        which = rng.choice([(True, False), (False, True), (True, True)])
        return _case(kind, sizes=sizes, parallel=which[0], delta=which[1], **step)
    return _case(kind, sizes=sizes, dtype=dtype, **step)


# ----------------------------------------------------------------------------- lengths of a step
def _lengths(case):
    """([tokens cached by each decoding entry], [(cached, new tokens) of each portion])."""
    rng = random.Random(f"{case['decoders']} {case['ctx_lo']} {case['ctx_hi']} {case['portions']} {case['rows']} {case['prior']}")
    ctx = [_log(rng, case["ctx_lo"], case["ctx_hi"]) for _ in range(case["decoders"])]  # tokens attended, the new one included
    n = case["portions"]
    weights = [rng.uniform(0.3, 1.7) for _ in range(n)]
    spare, rows = case["rows"] - n, []
    for i, w in enumerate(weights):
        part = spare if i == n - 1 else int(spare * w / sum(weights[i:]))
        rows.append(1 + part)
        spare -= part
    prior = [case["prior"] if i == 0 else (rng.randint(1, case["prior"]) if case["prior"] else 0) for i in range(n)]
    return [c - 1 for c in ctx], list(zip(prior, rows))


def _spans(case):
    """(first row, rows, tokens cached before) of every entry, decoding ones first."""
    decode, portions = _lengths(case)
    at, out = 0, []
    for cached, n in [(c, 1) for c in decode] + portions:
        out.append((at, n, cached))
        at += n
    return out


def _pairs(case, window=0):
    """(query, key) pairs that attention has to look at, and the tokens whose keys and values it needs."""
    pairs = seen = 0
    for _, n, cached in _spans(case):
        w = window or cached + n
        pairs += sum(min(p + 1, w) for p in range(cached, cached + n))
        seen += min(cached + n, n + w - 1)
    return pairs, seen


# ----------------------------------------------------------------------------- what a program has in hand
class _Random:
    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=self.gen, device=self.dev) * std).to(dtype)

    def uniform(self, *shape, lo, hi):
        return torch.rand(*shape, generator=self.gen, device=self.dev) * (hi - lo) + lo

    def weight(self, *shape):
        """A norm's weights, fp32."""
        return 1.0 + self.normal(*shape, std=0.1, dtype=torch.float32)


def _step(case, page, seed, dev):
    """The step's metadata on the device and the number of physical pages, in a random order."""
    decode, portions = _lengths(case)
    spans = _spans(case)
    n, entries = sum(s[1] for s in spans), len(spans)
    plan = S.plan_step(decode, portions, n, entries + 1)
    most = max((s[1] + s[2] + page - 1) // page for s in spans)
    table, pages = S.assign_pages(plan, page, most, torch.Generator().manual_seed(int(seed)))
    return S.upload_step(plan, table, [0] * n, dev), pages, n


def _rows(case, inp, n, slots=None):
    if case["portions"] == 0:
        B = case["decoders"]
        return ops.Rows(n, inp.cached_lens[:B], inp.num_decoding, inp.block_table[:B], slots=None if slots is None else slots[:B])
    return ops.Rows(n, inp.cached_lens, inp.num_decoding, inp.block_table, inp.seq_ids, inp.positions, inp.cu_seqlens, inp.tile_start,
                    inp.block_m, slots)


def _recorded(call, case):
    """`call` as a program keeps it: a graph to replay and its outputs, or the call itself."""
    if not case["graph"]:
        return {"call": call}
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    K.set_early_start(case["chained"])
    try:
        with torch.cuda.stream(s):
            call()
        torch.cuda.current_stream().wait_stream(s)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = call()
    finally:
        K.set_early_start(False)
    return {"graph": g, "out": out, "call": call}


def _int8_caches(r, case, pages):
    """Caches as earlier tokens left them: rows of normal values quantized to 8 bits, keys divided by their calibration."""
    caches = []
    for _ in range(case["layers"]):
        c = K.make_layer_cache(pages, S.HKV, case["page"], S.D, device=r.dev)
        for t in (c.k, c.v):
            flat = t.view(-1)
            for i in range(0, flat.numel(), 1 << 27):
                part = flat[i : i + (1 << 27)]
                part.copy_(torch.randn(part.numel(), generator=r.gen, device=r.dev).mul_(42.0).round_().clamp_(-127, 127))
        c.k_calibration.copy_(r.uniform(*c.k_calibration.shape, lo=1.5, hi=4.0))
        c.k_scale.copy_(r.uniform(*c.k_scale.shape, lo=0.006, hi=0.01))
        c.v_scale.copy_(r.uniform(*c.v_scale.shape, lo=0.018, hi=0.03))
        caches.append(c)
    return caches


def _int8_inputs(case, seed):
    r = _Random(seed)
    inp, pages, n = _step(case, case["page"], seed, r.dev)
    caches = _int8_caches(r, case, pages)
    width = (S.HQ + 2 * S.HKV) * S.D
    qkv = [r.normal(n, width, std=1.5) for _ in range(case["layers"])]
    qw, kw = ([r.weight(S.D).to(torch.bfloat16) for _ in range(case["layers"])] for _ in range(2))
    freq = S.ROPE_BASE ** (-torch.arange(0, S.D, 2, dtype=torch.float32, device=r.dev) / S.D)
    angle = inp.positions[:, None, None] * freq
    return inp, n, caches, qkv, qw, kw, angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)


def _prepare_int8(case, seed):
    inp, n, caches, qkv, qw, kw, cos, sin = _int8_inputs(case, seed)
    decoders, entries = case["decoders"], case["decoders"] + case["portions"]
    if not case["portions"]:
        step = HostDecodeStep(caches, decoders, S.HQ, S.HKV, S.D, tuple(inp.block_table[:decoders].shape), EPS)
        step.set_norm_weights(qw, kw)
        for dst, src in zip((step.dev_cos, step.dev_sin, step.dev_cached, step.dev_table, step.dev_nd),
                            (cos, sin, inp.cached_lens[:decoders], inp.block_table[:decoders], inp.num_decoding)):
            dst.copy_(src)
        step.dev_qkv.copy_(torch.stack(qkv))
        if case["graph"]:
            K.set_early_start(case["chained"])
            try:
                step.capture(groups=1)
            finally:
                K.set_early_start(False)
        return {"decode": step, "out": (step.dev_out, [_int8_state(c) for c in caches])}
    most = max(inp.prefix_tokens, 16)
    prefix_k = torch.empty(S.HKV, most, S.D, device=inp.ids.device, dtype=torch.bfloat16)
    prefix = S.PrefixScratch(prefix_k, torch.empty_like(prefix_k), inp.cu_cached)

    def call():
        plan = K.plan_decode_step(inp.cached_lens, inp.block_table, inp.num_decoding, caches[0])
        outs = []
        for i, cache in enumerate(caches):
            q, k, v = (t.view(n, -1, S.D) for t in qkv[i].split([S.HQ * S.D, S.HKV * S.D, S.HKV * S.D], dim=-1))
            outs.append(S.attention_ops(q, k, v, qw[i], kw[i], cos, sin, cache, inp, inp.cached_lens, inp.block_table, inp.num_decoding,
                                        prefix, plan))
        return outs, [_int8_state(c) for c in caches]

    return {"keep": (inp, prefix, entries), **_recorded(call, case)}


def _int8_state(c):
    return (c.k, c.v, c.k_scale, c.v_scale, c.k_calibration)


def _paged_inputs(case, seed):
    heads, kv, dim, vdim, rot = PAGED[case["sizes"]]
    r, dtype = _Random(seed), torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    inp, pages, n = _step(case, PAGE, seed, r.dev)
    cache = ops.make_paged_kv(pages, kv, PAGE, dim, vdim, dtype, r.dev)
    cache.k.normal_(generator=r.gen)  # keys have unit root mean square
    cache.v.normal_(generator=r.gen)
    qkv = r.normal(n, (heads + kv) * dim + kv * vdim, std=1.3, dtype=dtype)
    table = ops.Rotary(rot, 1e6).table(max(s[1] + s[2] for s in _spans(case)), r.dev)
    return inp, n, cache, qkv, table


def _prepare_paged(case, seed):
    heads, kv, dim, vdim, rot = PAGED[case["sizes"]]
    inp, n, cache, qkv, table = _paged_inputs(case, seed)
    rows = _rows(case, inp, n)

    def call():
        q = ops.rope_write(qkv, rows, cache, table, heads, True, True, EPS)
        return ops.paged_attention(q, cache, rows, dim ** -0.5), cache.k, cache.v

    return {"keep": inp, **_recorded(call, case)}


def _experts_inputs(case, seed):
    E, top, ff = EXPERTS[case["sizes"]]
    r, dtype = _Random(seed), torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    n = sum(s[1] for s in _spans(case))
    table = r.normal(VOCAB, WIDTH, dtype=dtype)
    ids = torch.randint(0, VOCAB, (n,), generator=r.gen, device=r.dev, dtype=torch.int32)
    # attention's output has a part that all rows share, so that some experts are chosen more often than others
    y = (r.normal(n, WIDTH, std=0.7, dtype=torch.float32) + r.normal(WIDTH, std=0.5, dtype=torch.float32)).to(dtype)
    norms = r.weight(WIDTH), r.weight(WIDTH)
    router = r.normal(E, WIDTH, std=0.03)
    gate, up = (r.normal(E, ff, WIDTH, std=0.03, dtype=dtype) for _ in range(2))
    down = r.normal(E, WIDTH, ff, std=0.03, dtype=dtype)
    return table, ids, y, norms, router, gate, up, down


def _prepare_experts(case, seed):
    E, top, ff = EXPERTS[case["sizes"]]
    table, ids, y, norms, router, gate, up, down = _experts_inputs(case, seed)
    dtype = table.dtype
    ex = ops.make_experts(router, gate, up, down, top, 7.0, GATE_SLOPE, dtype, table.device)

    def call():
        x, xb = ops.embed(table, ids)
        x, xb = ops.scaled_add_norm(x, y, norms[0], 2.0, EPS, dtype, zero=ex.counts)
        m, places = ops.mixture(x, xb, ex)
        return ops.scaled_add_norm(x, m, norms[1], 2.0, EPS, dtype, index=places)

    return _recorded(call, case)


def _parallel_inputs(r, case, inp, pages, n, slots):
    h, kv, d, vd, window, rot, sh, groups, state, p = PARALLEL[case["sizes"]]
    inner, bc = sh * p, groups * state
    cache = ops.make_paged_kv(pages, kv, PAGE, d, vd, torch.bfloat16, r.dev)
    cache.k.normal_(generator=r.gen)
    cache.v.normal_(generator=r.gen)
    parts = {"qkv": h * d + kv * (d + vd), "g": h, "z": inner, "xbc": inner + 2 * bc, "dt": sh}
    y = r.normal(n, sum(parts.values()))  # one product of the layer's input
    t = dict(zip(parts, y.split(list(parts.values()), dim=1)))
    norms = r.weight(h * d), r.weight(kv * d), r.weight(inner)
    dt_bias = torch.log(torch.expm1(torch.exp(r.uniform(sh, lo=math.log(1e-3), hi=math.log(0.1)))))
    rec = ops.Recurrence(sh, groups, state, p, r.normal(TAPS, inner + 2 * bc, std=0.5, dtype=torch.float32),
                         r.normal(inner + 2 * bc, std=0.1, dtype=torch.float32), -r.uniform(sh, lo=1.0, hi=16.0), dt_bias, r.weight(sh),
                         off_q=inner + bc, off_k=inner, off_v=0)
    sink = r.normal(h, dtype=torch.float32)
    table = ops.Rotary(rot, 1e6, stretch=2.0).table(max(s[1] + s[2] for s in _spans(case)), r.dev)
    return cache, t, norms, rec, sink, table, _state_inputs(r, rec, slots)


def _delta_inputs(r, case, n, slots):
    h, hk, d, vd = DELTA[case["sizes"]]
    qk, v = hk * d, h * vd
    parts = {"x": 2 * qk + v, "b": h, "step": h * d, "gate": v}
    t = {name: r.normal(n, size) for name, size in parts.items()}
    dt_bias = torch.log(torch.expm1(torch.exp(r.uniform(h * d, lo=math.log(1e-3), hi=math.log(0.1)))))
    rec = ops.Recurrence(h, hk, d, vd, r.normal(TAPS, 2 * qk + v, std=0.5, dtype=torch.float32), None, -r.uniform(h, lo=1.0, hi=16.0),
                         dt_bias, None, off_q=0, off_k=qk, off_v=2 * qk, channel_decay=True, correct=True, unit_eps=1e-6, q_scale=d ** -0.5)
    return t, r.weight(vd), rec, _state_inputs(r, rec, slots)


def _state_inputs(r, rec, slots):
    """States and the convolution's last inputs as earlier tokens left them."""
    return r.normal(slots, rec.heads, rec.dim, rec.vdim, std=0.3, dtype=torch.float32), r.normal(slots, rec.taps, rec.channels)


def _parallel(r, case, inp, pages, n, rows):
    """(one layer's call, [(buffer, what earlier tokens left in it)])."""
    h, kv, d, vd, window, rot, sh, groups, state, p = PARALLEL[case["sizes"]]
    entries = case["decoders"] + case["portions"]
    cache, t, norms, rec, sink, table, first = _parallel_inputs(r, case, inp, pages, n, entries)
    st = ops.make_recurrent_state(rec, entries, torch.bfloat16, r.dev)
    gated = ops.GatedNorm(norms[2], groups, EPS, gate_first=True, out_scale=0.7)

    def call():
        both = torch.empty(n, h * vd + sh * p, dtype=torch.bfloat16, device=r.dev)
        q = ops.norm_rope_write(t["qkv"], rows, cache, norms[0], norms[1], EPS, table, h)
        ops.paged_attention(q, cache, rows, d ** -0.5, ops.AttnOptions(window, sink, t["g"], 0.8), both[:, : h * vd].unflatten(1, (h, vd)))
        ops.recurrent_mixer(rec, st, t["xbc"], t["dt"], None, t["z"], gated, rows, both[:, h * vd :])
        return both, cache.k, cache.v, st.state, st.ring

    return call, [(st.state, first[0]), (st.ring, first[1])]


def _delta(r, case, n, rows):
    h, hk, d, vd = DELTA[case["sizes"]]
    entries = case["decoders"] + case["portions"]
    t, weight, rec, first = _delta_inputs(r, case, n, entries)
    st = ops.make_recurrent_state(rec, entries, torch.bfloat16, r.dev)
    norm = ops.GatedNorm(weight, h, EPS, gate_first=False)

    def call():
        o = torch.empty(n, h * vd, dtype=torch.bfloat16, device=r.dev)
        ops.recurrent_mixer(rec, st, t["x"], t["step"], t["b"], t["gate"], norm, rows, o)
        return o, st.state, st.ring

    return call, [(st.state, first[0]), (st.ring, first[1])]


def _prepare_state(case, seed):
    r = _Random(seed)
    inp, pages, n = _step(case, PAGE, seed, r.dev)
    entries = case["decoders"] + case["portions"]
    slots = torch.cat([torch.randperm(entries, generator=r.gen, device=r.dev), torch.tensor([-1], device=r.dev)]).to(torch.int32)
    rows = _rows(case, inp, n, slots)
    layers = []
    if case["parallel"]:
        layers.append(_parallel(r, case, inp, pages, n, rows))
    if case["delta"]:
        layers.append(_delta(r, case, n, rows))
    kept = _recorded(lambda: [call() for call, _ in layers], case)
    for dst, src in [x for _, fill in layers for x in fill]:  # after the recording, whose warm-up advances the states
        dst.copy_(src)
    return {"keep": (inp, slots), **kept}


def prepare(case, seed):
    kinds = {"int8": _prepare_int8, "paged": _prepare_paged, "experts": _prepare_experts, "state": _prepare_state}
    with torch.inference_mode():
        return kinds[case["kind"]](case, seed)


def run(state):
    if "decode" in state:
        state["decode"].run_device()
        return state["out"]
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    with torch.inference_mode():
        return state["call"]()


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    n = sum(s[1] for s in _spans(case))
    size = 4 if case.get("dtype") == "fp32" else 2
    if case["kind"] == "int8":
        pairs, seen = _pairs(case)
        token = 2 * S.HKV * (S.D + 4)
        row = (S.HQ + 2 * S.HKV) * S.D * 2 + S.HQ * S.D * 2
        return {"bytes": case["layers"] * (seen * token + n * row), "flops": case["layers"] * 4 * S.D * S.HQ * pairs}
    if case["kind"] == "paged":
        heads, kv, dim, vdim, _ = PAGED[case["sizes"]]
        pairs, seen = _pairs(case)
        row = (heads + kv) * dim + kv * vdim + heads * vdim
        return {"bytes": size * (seen * kv * (dim + vdim) + n * row), "flops": 2 * (dim + vdim) * heads * pairs}
    if case["kind"] == "experts":
        E, top, ff = EXPERTS[case["sizes"]]
        used = min(E, n * top)
        return {"bytes": size * (used * 3 * ff * WIDTH + 3 * n * WIDTH) + E * WIDTH * 2 + 4 * n * WIDTH, "flops": 6 * n * top * ff * WIDTH}
    total = {"bytes": 0, "flops": 0}
    entries = case["decoders"] + case["portions"]
    if case["parallel"]:
        h, kv, d, vd, window, _, sh, groups, state, p = PARALLEL[case["sizes"]]
        pairs, seen = _pairs(case, window)
        row = h * d + kv * (d + vd) + h + 2 * sh * p + 2 * groups * state + sh + h * vd + sh * p
        total["bytes"] += 2 * (seen * kv * (d + vd) + n * row) + 8 * entries * sh * state * p
        total["flops"] += 2 * (d + vd) * h * pairs + 4 * n * sh * state * p
    if case["delta"]:
        h, hk, d, vd = DELTA[case["sizes"]]
        total["bytes"] += 2 * n * (2 * hk * d + h * vd + h + h * d + 2 * h * vd) + 8 * entries * h * d * vd
        total["flops"] += 8 * n * h * d * vd
    return total


def tolerance(case):
    if case["kind"] != "int8" and case.get("dtype") == "fp32":
        return {"rel": 2e-6, "max": 1e-4}
    if case["kind"] == "int8":  # codes of rows that are rounded to bf16 first fall beside one another now and then
        return {"rel": 1e-2, "max": 0.2, "differ": 1e-3}
    return {"rel": 1e-2, "max": 0.2}


# ----------------------------------------------------------------------------- the same in 64 bits
def _attend(q, k, v, cached, scale, window=0, sink=None):
    """q [n, H, d] at positions cached.., k [S, G, d], v [S, G, vd] from position 0 -> [n, H, vd]."""
    n, H, _ = q.shape
    G = k.shape[1]
    pos = cached + torch.arange(n, device=q.device)[:, None]
    key = torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = key > pos
    if window:
        hidden = hidden | (key <= pos - window)
    out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T * scale).masked_fill(hidden, -math.inf)
        top = s.amax(dim=1, keepdim=True)
        if sink is not None:
            top = top.clamp(min=float(sink[h]))
        p = torch.exp(s - top)
        den = p.sum(dim=1, keepdim=True)
        if sink is not None:
            den = den + torch.exp(sink[h] - top)
        out[:, h] = (p / den) @ v[:, h // (H // G)]
    return out


def _rms(x, weight=None):
    y = x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + EPS)
    return y if weight is None else y * weight


def _at(table, entry, first, last, page):
    """(physical page, row of it) of an entry's tokens first .. last - 1."""
    t = torch.arange(first, last, device=table.device)
    return table[entry].long()[t // page], t % page


def _quantized(x):
    scale = x.abs().amax(dim=-1).clamp(min=1e-6) / 127
    return torch.round(x / scale[..., None]).clamp(-127, 127) * scale[..., None], scale


def _exact_int8(case, seed):
    inp, n, caches, qkv, qw, kw, cos, sin = _int8_inputs(case, seed)
    c, s = cos.double(), sin.double()
    half = S.D // 2
    page, outs, states = case["page"], [], []

    def normed(x, w):
        y = _rms(x, w.double())
        a, b = y[..., :half], y[..., half:]
        return torch.cat([a * c - b * s, a * s + b * c], dim=-1)

    for i, cache in enumerate(caches):
        q, k, v = (t.double().view(n, -1, S.D) for t in qkv[i].split([S.HQ * S.D, S.HKV * S.D, S.HKV * S.D], dim=-1))
        q, k = normed(q, qw[i]), normed(k, kw[i])
        out = torch.empty(n, S.HQ, S.D, dtype=torch.float64, device=q.device)
        ks, vs, cal = cache.k_scale.double(), cache.v_scale.double(), cache.k_calibration.double()
        for e, (at, m, cached) in enumerate(_spans(case)):
            first = inp.block_table[e, 0].long()
            new_k, new_v = k[at : at + m], v[at : at + m]
            prompt = e >= case["decoders"]
            if prompt and cached == 0:
                cal[first, :, 0] = new_k.abs().amax(dim=0).clamp(min=1e-3)
            mine = cal[first, :, 0]
            kq, k_sc = _quantized(new_k / mine)
            vq, v_sc = _quantized(new_v)
            pg, row = _at(inp.block_table, e, 0, cached, page)
            old_k = cache.k[pg, :, row].double() * ks[pg, :, row][..., None] * mine
            old_v = cache.v[pg, :, row].double() * vs[pg, :, row][..., None]
            pg, row = _at(inp.block_table, e, cached, cached + m, page)
            ks[pg, :, row], vs[pg, :, row] = k_sc, v_sc
            # a portion's own rows are attended as they are, a decoded token as the cache holds it
            seen_k, seen_v = (new_k, new_v) if prompt else (kq * mine, vq)
            out[at : at + m] = _attend(q[at : at + m], torch.cat([old_k, seen_k]), torch.cat([old_v, seen_v]), cached, S.D ** -0.5)
        outs.append(out)
        states.append((None, None, ks, vs, cal))
    return (outs if case["portions"] else torch.stack(outs)), states


def _exact_attention(case, inp, cache, q, k, v, scale, window=0, sink=None):
    """Attention of every entry over its cached tokens and the step's own; the cache with these in it."""
    ck, cv = cache.k.double(), cache.v.double()
    d, vd = cache.k_dim, cache.v_dim
    out = torch.empty(q.shape[0], q.shape[1], vd, dtype=torch.float64, device=q.device)
    for e, (at, m, cached) in enumerate(_spans(case)):
        pg, row = _at(inp.block_table, e, cached, cached + m, cache.page_size)
        ck[pg, :, row, :d], cv[pg, :, row, :vd] = k[at : at + m], v[at : at + m]
        pg, row = _at(inp.block_table, e, 0, cached + m, cache.page_size)
        out[at : at + m] = _attend(q[at : at + m], ck[pg, :, row, :d], cv[pg, :, row, :vd], cached, scale, window, sink)
    return out, ck, cv


def _exact_paged(case, seed):
    heads, kv, dim, vdim, rot = PAGED[case["sizes"]]
    inp, n, cache, qkv, _ = _paged_inputs(case, seed)
    q, k, v = qkv.double().split([heads * dim, kv * dim, kv * vdim], dim=1)
    angle = inp.positions[:, None, None].double() * 1e6 ** (-2.0 * torch.arange(rot // 2, device=q.device, dtype=torch.float64) / rot)

    def turned(x):
        x = x.reshape(n, -1, dim)
        a, b = x[..., : rot // 2], x[..., rot // 2 : rot]
        return _rms(torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), x[..., rot:]], dim=-1))

    return _exact_attention(case, inp, cache, turned(q), turned(k), v.reshape(n, kv, vdim), dim ** -0.5)


def _exact_experts(case, seed):
    E, top, ff = EXPERTS[case["sizes"]]
    table, ids, y, norms, router, gate, up, down = _experts_inputs(case, seed)
    x = _rms(2.0 * table[ids.long()].double() + y.double(), norms[0].double())
    scores, chosen = torch.sigmoid(x @ router.double().T).topk(top, dim=1)
    out = torch.zeros_like(x)
    for e in range(E):
        t, place = (chosen == e).nonzero(as_tuple=True)
        if len(t) == 0:
            continue
        h = x[t] * scores[t, place][:, None]
        g, u = (h @ gate[e].double().T).clamp(max=7.0), (h @ up[e].double().T).clamp(-7.0, 7.0)
        out.index_add_(0, t, (g * torch.sigmoid(GATE_SLOPE * g) * (u + 1.0)) @ down[e].double().T)
    x = _rms(2.0 * x + out, norms[1].double())
    return x, x


def _exact_recurrence(case, rec, x, step, beta, first, slots):
    """Convolution, state and read-out of every entry, token by token: (o [n, heads, vdim], states, rings)."""
    n, per = x.shape[0], rec.heads // rec.qk_heads
    state, ring = first[0].double(), first[1].double()
    x, w = x.double(), rec.conv_w.double()
    wide = rec.heads * (rec.dim if rec.channel_decay else 1)
    neg_a = rec.neg_a.double().repeat_interleave(wide // rec.heads)
    grow = torch.nn.functional.softplus(step.double() + rec.dt_bias.double(), threshold=1e9)
    decay = torch.exp(neg_a * grow).view(n, rec.heads, -1, 1)
    out = torch.empty(n, rec.heads, rec.vdim, dtype=torch.float64, device=x.device)
    for e, (at, m, cached) in enumerate(_spans(case)):
        slot = int(slots[e])
        before = [ring[slot, p % rec.taps] if p >= 0 else torch.zeros_like(x[0]) for p in range(cached - rec.taps + 1, cached)]
        ext = torch.cat([torch.stack(before), x[at : at + m]])
        y = sum(ext[j : j + m] * w[j] for j in range(rec.taps))
        y = torch.nn.functional.silu(y if rec.conv_b is None else y + rec.conv_b.double())
        q = y[:, rec.off_q : rec.off_q + rec.qk_heads * rec.dim].view(m, rec.qk_heads, rec.dim)
        k = y[:, rec.off_k : rec.off_k + rec.qk_heads * rec.dim].view(m, rec.qk_heads, rec.dim)
        v = y[:, rec.off_v : rec.off_v + rec.heads * rec.vdim].view(m, rec.heads, rec.vdim)
        if rec.unit_eps is not None:
            q, k = (t / torch.sqrt((t * t).sum(dim=-1, keepdim=True) + rec.unit_eps) for t in (q, k))
        q, k = (t.repeat_interleave(per, dim=1) for t in (q * rec.q_scale, k))
        s = state[slot] if cached else torch.zeros_like(state[slot])
        for t in range(m):
            s = s * decay[at + t]
            if rec.correct:
                u = torch.sigmoid(beta[at + t].double())[:, None] * (v[t] - (k[t][:, None] @ s)[:, 0])
            else:
                u = grow[at + t][:, None] * v[t]
            s = s + k[t][:, :, None] * u[:, None]
            out[at + t] = (q[t][:, None] @ s)[:, 0]
        if rec.skip is not None:
            out[at : at + m] += rec.skip.double()[:, None] * v
        state[slot] = s
        for t in range(max(0, m - rec.taps), m):
            ring[slot, (cached + t) % rec.taps] = x[at + t]
    return out, state, ring


def _exact_state(case, seed):
    r = _Random(seed)
    inp, pages, n = _step(case, PAGE, seed, r.dev)
    entries = case["decoders"] + case["portions"]
    slots = torch.randperm(entries, generator=r.gen, device=r.dev).tolist()
    res = []
    if case["parallel"]:
        h, kv, d, vd, window, rot, sh, groups, state, p = PARALLEL[case["sizes"]]
        cache, t, norms, rec, sink, _, first = _parallel_inputs(r, case, inp, pages, n, entries)
        q, k, v = t["qkv"].double().split([h * d, kv * d, kv * vd], dim=1)
        angle = inp.positions[:, None, None].double() * (1e6 ** (-2.0 * torch.arange(rot // 2, device=r.dev, dtype=torch.float64) / rot) / 2.0)

        def turned(x):
            x = x.reshape(n, -1, d)
            a, b = x[..., 0:rot:2], x[..., 1:rot:2]
            pair = torch.stack([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1).flatten(-2)
            return torch.cat([pair, x[..., rot:]], dim=-1)

        q, k = turned(_rms(q, norms[0].double())), turned(_rms(k, norms[1].double()))
        a, ck, cv = _exact_attention(case, inp, cache, q, k, v.reshape(n, kv, vd), d ** -0.5, window, sink.double())
        a = 0.8 * a * torch.sigmoid(t["g"].double())[:, :, None]
        o, st, ring = _exact_recurrence(case, rec, t["xbc"], t["dt"], None, first, slots)
        o = o.reshape(n, -1) * torch.nn.functional.silu(t["z"].double())
        o = 0.7 * _rms(o.view(n, groups, -1)).reshape(n, -1) * norms[2].double()
        res.append((torch.cat([a.reshape(n, -1), o], dim=1), ck, cv, st, ring))
    if case["delta"]:
        t, weight, rec, first = _delta_inputs(r, case, n, entries)
        o, st, ring = _exact_recurrence(case, rec, t["x"], t["step"], t["b"], first, slots)
        o = _rms(o, weight.double()).reshape(n, -1) * torch.sigmoid(t["gate"].double())
        res.append((o, st, ring))
    return res


def exact(case, seed):
    kinds = {"int8": _exact_int8, "paged": _exact_paged, "experts": _exact_experts, "state": _exact_state}
    with torch.inference_mode():
        return kinds[case["kind"]](case, seed)
