"""Steps with portions recorded into a CUDA graph, where portions, decoding entries and the fetch of cached tokens are branches beside one
another: replayed on changed inputs, outputs and scratch poisoned in between, bit for bit what the calls give in order."""
import numpy as np
import pytest
import torch

from tests import helpers as H
from tests.helpers import D, HKV, HQ

pytestmark = pytest.mark.gpu
DEV = "cuda"
# tokens cached by each decoding entry, (cached, new) of each portion: decoding beside first and continued portions, either alone, many of both
STEPS = [([37, 130], [(48, 70), (0, 33)]), ([], [(0, 90), (200, 50), (0, 1)]), ([5], [(300, 257)]), ([700, 64, 15, 2000], [(0, 64), (16, 20), (1000, 130)])]


def recorded(call, chained):
    """(graph, its outputs) of `call`, run once before as every recording is."""
    from inference_engine_b200 import kernels as K

    K.set_early_start(chained)
    try:
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            call()
        torch.cuda.current_stream().wait_stream(s)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = call()
    finally:
        K.set_early_start(False)
    return graph, out


def step_of(decode, portions, page):
    from inference_engine_b200 import scaffold as S

    n = len(decode) + sum(x for _, x in portions) + 7  # a padding entry of seven rows
    plan = S.plan_step(decode, portions, n, len(decode) + len(portions) + 3)
    table, pages = S.assign_pages(plan, page, max(-(-(c + x) // page) for c, x in [(c, 1) for c in decode] + portions + [(0, 7)]),
                                  torch.Generator().manual_seed(3))
    return S.upload_step(plan, table, [0] * n, DEV), pages, n


@pytest.mark.parametrize("chained", [False, True])
@pytest.mark.parametrize("decode,portions", STEPS)
def test_int8_steps(decode, portions, chained):
    from inference_engine_b200 import kernels as K
    from inference_engine_b200 import scaffold as S

    inp, pages, n = step_of(decode, portions, 16)
    g = torch.Generator(device=DEV).manual_seed(n)
    filled = [H.cache_to_torch(H.random_filled_cache(np.random.default_rng(i), pages, 16, gauss=True)) for i in range(2)]
    caches = [H.cache_to_torch(H.random_filled_cache(np.random.default_rng(9), pages, 16, gauss=True)) for _ in range(2)]
    parts = lambda c: (c.k, c.v, c.k_scale, c.v_scale, c.k_calibration)
    qkv = [torch.randn(n, HQ + 2 * HKV, D, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2)]
    qw, kw = (1 + 0.1 * torch.randn(D, generator=g, device=DEV)).to(torch.bfloat16), torch.ones(D, device=DEV, dtype=torch.bfloat16)
    angle = torch.rand(n, 1, D // 2, generator=g, device=DEV) * 6
    cos, sin = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)
    scratch = [torch.empty(HKV, inp.prefix_tokens + 8, D, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    prefix = S.PrefixScratch(*scratch, inp.cu_cached)

    def call():
        plan = K.plan_decode_step(inp.cached_lens, inp.block_table, inp.num_decoding, caches[0])
        return [S.attention_ops(*x.split([HQ, HKV, HKV], dim=1), qw, kw, cos, sin, c, inp, inp.cached_lens, inp.block_table, inp.num_decoding,
                                prefix, plan) for x, c in zip(qkv, caches)]

    def start_over():
        for c, f in zip(caches, filled):
            for dst, src in zip(parts(c), parts(f)):
                dst.copy_(src)
        for t in scratch:
            t.fill_(float("nan"))

    graph, outs = recorded(call, chained)
    for _ in range(3):
        for x in qkv:
            x.normal_(generator=g)
        start_over()
        want = [o.clone() for o in call()]
        want_caches = [[t.clone() for t in parts(c)] for c in caches]
        start_over()
        for o in outs:
            o.fill_(float("nan"))
        graph.replay()
        for o, w in zip(outs, want):
            assert torch.equal(o, w) and not o.isnan().any()
        for c, w in zip(caches, want_caches):
            assert all(torch.equal(a, b) for a, b in zip(parts(c), w))
    assert K.check_status() == 0


@pytest.mark.parametrize("chained", [False, True])
@pytest.mark.parametrize("heads,kv,dim,vdim,window", [(16, 8, 128, 128, 0), (16, 4, 64, 48, 100)])
@pytest.mark.parametrize("decode,portions", STEPS)
def test_paged_steps(decode, portions, heads, kv, dim, vdim, window, chained):
    from inference_engine_b200 import kernels as K
    from inference_engine_b200 import ops

    inp, pages, n = step_of(decode, portions, 16)
    g = torch.Generator(device=DEV).manual_seed(n)
    filled, caches = ([ops.make_paged_kv(pages, kv, 16, dim, vdim, torch.bfloat16, DEV) for _ in range(2)] for _ in range(2))
    for c in filled:
        c.k[..., :dim].normal_(generator=g)
        c.v[..., :vdim].normal_(generator=g)
    qkv = [torch.randn(n, heads * dim + kv * (dim + vdim), generator=g, device=DEV).to(torch.bfloat16) for _ in range(2)]
    table = ops.Rotary(dim, 1e4).table(4096, DEV)
    rows = ops.Rows(n, inp.cached_lens, inp.num_decoding, inp.block_table, inp.seq_ids, inp.positions, inp.cu_seqlens, inp.tile_start, inp.block_m)
    opt = ops.AttnOptions(window=window, sink=torch.randn(heads, generator=g, device=DEV)) if window else None

    def call():
        return [ops.paged_attention(ops.rope_write(x, rows, c, table, heads, True, True, 1e-6), c, rows, dim ** -0.5, opt) for x, c in zip(qkv, caches)]

    def start_over():
        for c, f in zip(caches, filled):
            c.k.copy_(f.k)
            c.v.copy_(f.v)

    graph, outs = recorded(call, chained)
    for _ in range(3):
        for x in qkv:
            x.normal_(generator=g)
        start_over()
        want = [o.clone() for o in call()]
        want_caches = [(c.k.clone(), c.v.clone()) for c in caches]
        start_over()
        for o in outs:
            o.fill_(float("nan"))
        graph.replay()
        for o, w in zip(outs, want):
            assert torch.equal(o, w) and not o.isnan().any()
        for c, (k, v) in zip(caches, want_caches):
            assert torch.equal(c.k, k) and torch.equal(c.v, v)
    assert K.check_status() == 0
