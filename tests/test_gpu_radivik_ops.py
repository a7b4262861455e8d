"""Each mechanism of the decoder ops alone, against the plain implementation."""
import numpy as np
import pytest
import torch

from oracle import radivik as R
from tests import radivik_helpers as H

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]
DEV = "cuda"


def t(x, dtype=torch.float32):
    return torch.as_tensor(np.asarray(x, np.float32)).to(dtype).to(DEV)


def i32(x):
    return torch.as_tensor(np.asarray(x, np.int32)).to(DEV)


def close(got, want, dtype, tol=None):
    got, want = got.detach().float().cpu().numpy(), np.asarray(want)
    tol = tol or (3e-6 if dtype == torch.float32 else 1e-2)
    err = np.abs(got - want).max() / max(1.0, np.abs(want).max())
    assert err < tol, err


def make_rows(entries, page=16, pages_extra=3, seed=0):
    """entries: [(cached, new)]; decoding ones (new == 1 and cached > 0) first.  A scattered block table."""
    from inference_engine_b200 import ops
    from inference_engine_b200.scaffold import plan_step

    nd = 0
    while nd < len(entries) and entries[nd][1] == 1 and entries[nd][0] > 0:
        nd += 1
    n = sum(x for _, x in entries)
    plan = plan_step([c for c, _ in entries[:nd]], entries[nd:], n, len(entries) + 1)
    need = [(c + x + page - 1) // page for c, x in entries]
    perm = np.random.default_rng(seed).permutation(sum(need) + pages_extra)
    table = np.full((len(entries) + 1, max(need)), -1, np.int32)
    at = 0
    for b, k in enumerate(need):
        table[b, :k] = perm[at : at + k]
        at += k
    rows = ops.Rows(n, i32(plan["cached"]), i32([nd]), i32(table), i32(plan["seq_ids"]), i32(plan["positions"]), i32(plan["cu_seqlens"]),
                    i32(plan["tile_start"]), 128)
    return rows, table, len(perm), plan


def fill(cache, table, b, k, v):
    """Place keys [n, heads, dim] and values of an entry in the cache by its pages."""
    P = cache.page_size
    for j in range(k.shape[0]):
        cache.k[int(table[b, j // P]), :, j % P, : k.shape[2]] = k[j]
        cache.v[int(table[b, j // P]), :, j % P, : v.shape[2]] = v[j]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,top", [(64, 1), (2052, 3), (33, 2)])
def test_scaled_add_norm(dtype, width, top):
    from inference_engine_b200 import ops

    g = np.random.default_rng(1)
    x, w = g.standard_normal((7, width)), H.bf16(1 + 0.3 * g.standard_normal(width))
    d = H.bf16(g.standard_normal((7 * top, width)))
    index = g.permutation(7 * top).reshape(7, top)
    want = R.rms_norm(2.25 * np.float32(x) + d[index].sum(1), 1e-3, w)
    zero = torch.ones(5, dtype=torch.int32, device=DEV)
    y, yb = ops.scaled_add_norm(t(x), t(d, dtype), t(w), 2.25, 1e-3, dtype, index=i32(index), zero=zero)
    close(y, want, torch.float32)
    close(yb, want, dtype)
    assert zero.sum().item() == 0
    x0 = t(x)
    _, only = ops.scaled_add_norm(x0, None, t(w), 1.0, 1e-3, dtype, keep=False)
    close(only, R.rms_norm(np.float32(x), 1e-3, w), dtype)
    close(x0, x, torch.float32)  # untouched


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,top", [(2048, 4), (1028, 5), (64, 9), (4096, 3)])
def test_scaled_add_norm_of_several_experts(dtype, width, top):
    """Rows of a token's experts that are fetched together, and more of them than are."""
    test_scaled_add_norm(dtype, width, top)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("scaling", [None, H.YARN])
@pytest.mark.parametrize("dim,vdim,rot", [(48, 40, 16), (20, 36, 20), (7, 130, 2)])
def test_rotation_unit_norm_and_write(dtype, scaling, dim, vdim, rot):
    from inference_engine_b200 import ops

    g = np.random.default_rng(2)
    heads, kv, eps = 4, 2, 1e-4
    rows, table, pages, plan = make_rows([(33, 1), (15, 1), (0, 5), (14, 40)])
    cache = ops.make_paged_kv(pages, kv, 16, dim, vdim, dtype, DEV)
    rd = {"dims": rot, "base": 500.0, **({"scaling": scaling} if scaling else {})}
    rotary = ops.Rotary(rot, 500.0, None if not scaling else tuple(float(scaling[k]) for k in ("factor", "original", "fast", "slow")))
    f, mult = R.rotary_frequencies(rd)
    assert np.allclose(rotary.frequencies()[0], f, rtol=1e-12) and rotary.frequencies()[1] == mult
    qkv = H.bf16(g.standard_normal((rows.num_rows, (heads + kv) * dim + kv * vdim)))
    q = ops.rope_write(t(qkv, dtype), rows, cache, rotary.table(64, DEV), heads, True, True, eps)
    pos, seq = np.array(plan["positions"]), np.array(plan["seq_ids"])
    n = rows.num_rows
    close(q[..., :dim], R.rms_norm(R.rotate(qkv[:, : heads * dim].reshape(n, heads, dim), pos, rd), eps), dtype)
    assert q[..., dim:].abs().sum().item() == 0
    k = R.rms_norm(R.rotate(qkv[:, heads * dim : (heads + kv) * dim].reshape(n, kv, dim), pos, rd), eps)
    v = qkv[:, (heads + kv) * dim :].reshape(n, kv, vdim)
    page, slot = table[seq, pos // 16], pos % 16
    close(cache.k[page, :, slot][..., :dim], k, dtype)
    close(cache.v[page, :, slot][..., :vdim], v, dtype)
    touched = np.zeros((pages, 16), bool)
    touched[page, slot] = True
    assert cache.k.permute(0, 2, 1, 3)[torch.as_tensor(~touched)].abs().sum().item() == 0  # nothing else was written
    # queries only: the cache stays as it is
    before = cache.k.clone()
    q2 = ops.rope_write(t(qkv[:, : heads * dim], dtype), rows, cache, rotary.table(64, DEV), heads, False, True, eps)
    assert torch.equal(q, q2) and torch.equal(before, cache.k)
    H.status_clear()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("dim,vdim,rot", [(112, 96, 32), (128, 128, 128), (64, 8, 48), (8, 64, 0), (16, 16, 16)])
def test_rotation_by_whole_rows(dtype, dim, vdim, rot):
    """Sizes in eights: eight and sixteen lanes a head, heads that leave lanes idle, a rotation of all, some and none of the channels."""
    if rot:
        test_rotation_unit_norm_and_write(dtype, None, dim, vdim, rot)
    from inference_engine_b200 import ops

    g = np.random.default_rng(dim)
    heads, kv, n = 6, 3, 1300  # enough rows for few threads and several heads each; one page of one row per entry
    cache = ops.make_paged_kv(n, kv, 16, dim, vdim, dtype, DEV)
    perm = g.permutation(n)
    rows = ops.Rows(n, i32(np.zeros(n)), i32([n - 2]), i32(perm[:, None]))  # a decode step with two idle rows
    qkv = H.bf16(g.standard_normal((n, (heads + kv) * dim + kv * vdim)))
    table = ops.Rotary(rot, 500.0).table(4, DEV) if rot else None
    q = ops.rope_write(t(qkv, dtype), rows, cache, table, heads, True, False, 1e-4)
    live = slice(0, n - 2)
    close(q[live, :, :dim], qkv[live, : heads * dim].reshape(-1, heads, dim), dtype)
    assert q[n - 2 :].abs().sum().item() == 0
    close(cache.k[perm[live], :, 0, :dim], qkv[live, heads * dim : (heads + kv) * dim].reshape(-1, kv, dim), dtype)
    close(cache.v[perm[live], :, 0, :vdim], qkv[live, (heads + kv) * dim :].reshape(-1, kv, vdim), dtype)
    H.status_clear()


CASES = [  # heads, kv heads, key size, value size
    (4, 2, 48, 40), (3, 1, 128, 64), (8, 8, 64, 128), (12, 1, 104, 88), (40, 2, 16, 24), (2, 1, 36, 12), (2, 2, 10, 7),
]


@pytest.mark.parametrize("heads,kv,dim,vdim", CASES)
@pytest.mark.parametrize("page", [16, 64])
def test_attention_single_key_stands_out(heads, kv, dim, vdim, page):
    """Every query matches one key far above all others (its own position, the first key, both sides of page and block
    borders, the key just outside the causal edge as a decoy), in prompt portions and decoding rows of one step."""
    from inference_engine_b200 import ops

    g = np.random.default_rng(3)
    entries = [(16, 1), (63, 1), (64, 1), (700, 1), (0, 130), (61, 67), (257, 2)]
    rows, table, pages, plan = make_rows(entries, page)
    cache = ops.make_paged_kv(pages, kv, page, dim, vdim, torch.bfloat16, DEV)
    cache.k.fill_(float("nan"))  # whatever no token was written to must not matter
    cache.v.fill_(float("nan"))
    cache.k[..., dim:] = 0
    cache.v[..., vdim:] = 0
    q = np.zeros((rows.num_rows, heads, dim))
    want = np.zeros((rows.num_rows, heads, vdim))
    at = 0
    scale = 24.0 / np.sqrt(dim)
    for b, (c, x) in enumerate(entries):
        n = c + x
        k = H.bf16(R.rms_norm(g.standard_normal((n, kv, dim)), 1e-6))
        v = H.bf16(g.standard_normal((n, kv, vdim)))
        fill(cache, table, b, t(k, torch.bfloat16), t(v, torch.bfloat16))
        for i in range(x):
            p = c + i
            targets = [p, 0, max(0, p - 1), min(p, 15), min(p, 16), min(p, 63), min(p, 64), p // 64 * 64, min(n - 1, p + 1)]
            for h in range(heads):
                q[at + i, h] = k[targets[(i + h) % len(targets)], h // (heads // kv)]
        q[at : at + x] = H.bf16(q[at : at + x])
        want[at : at + x] = R.causal_attention(q[at : at + x], k, v, scale, c)
        at += x
    qd = torch.zeros(rows.num_rows, heads, cache.k.shape[3], device=DEV, dtype=torch.bfloat16)
    qd[..., :dim] = t(q, torch.bfloat16)
    close(ops.attention_rows(qd, cache, rows, scale), want, torch.bfloat16)
    assert ops.tensor_core_attention(cache)
    for _ in range(2):  # the second call finds the workspace as the first left it
        close(ops.paged_attention(qd, cache, rows, scale), want, torch.bfloat16, 2e-2)
    H.status_clear()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv,dim,vdim", [(2, 2, 24, 40), (16, 1, 32, 132), (5, 1, 36, 256), (34, 2, 16, 8), (4, 2, 184, 184), (4, 2, 192, 192)])
def test_attention_rows_in_tiles(heads, kv, dim, vdim, dtype):
    """Tiles of neighbouring rows at their edges: groups of 1 to 17 query heads, entries that begin and end within a tile or
    one key around a step of 64, the largest sizes of the tiles and the first beyond; a row's result does not depend on what
    a later token's key and value are."""
    from inference_engine_b200 import ops

    g = np.random.default_rng(dim)
    entries = [(63, 1), (500, 1), (0, 66), (61, 7), (64, 64), (125, 5), (7, 1)]
    rows, table, pages, _ = make_rows(entries, 8)
    cache = ops.make_paged_kv(pages, kv, 8, dim, vdim, dtype, DEV)
    q, want, at = H.bf16(g.standard_normal((rows.num_rows, heads, dim))), np.zeros((rows.num_rows, heads, vdim)), 0
    ends = []
    for b, (c, x) in enumerate(entries):
        k, v = H.bf16(g.standard_normal((c + x, kv, dim))), H.bf16(g.standard_normal((c + x, kv, vdim)))
        fill(cache, table, b, t(k, dtype), t(v, dtype))
        want[at : at + x] = R.causal_attention(q[at : at + x], k, v, dim ** -0.5, c)
        at += x
        ends.append((at - 1, int(table[b, (c + x - 1) // 8]), (c + x - 1) % 8))
    qd = torch.zeros(rows.num_rows, heads, cache.k.shape[3], device=DEV, dtype=dtype)
    qd[..., :dim] = t(q, dtype)
    out = ops.attention_rows(qd, cache, rows, dim ** -0.5)
    close(out, want, dtype)
    for _, page, slot in ends:
        cache.k[page, :, slot], cache.v[page, :, slot] = float("nan"), float("inf")
    again = ops.attention_rows(qd, cache, rows, dim ** -0.5)
    others = [r for r in range(rows.num_rows) if r not in [e[0] for e in ends]]
    assert torch.equal(out[others], again[others])
    H.status_clear()


@pytest.mark.parametrize("heads,kv,dim,vdim,window", [(16, 8, 128, 128, 0), (15, 5, 64, 48, 0), (15, 3, 48, 40, 100)])
@pytest.mark.parametrize("entries", [[(0, 1), (0, 1200)], [(0, 700), (200, 129), (40, 515)], [(0, 65)] * 20, [(700, 40)] * 12])
def test_prompt_attention_of_many_tiles(heads, kv, dim, vdim, window, entries):
    """More tiles and heads than multiprocessors: two heads a block where a tile has few keys, also an odd number of heads, beside tiles with more."""
    from inference_engine_b200 import ops

    g = np.random.default_rng(heads + len(entries))
    rows, table, pages, _ = make_rows(entries, 16)
    cache = ops.make_paged_kv(pages, kv, 16, dim, vdim, torch.bfloat16, DEV)
    cache.k.fill_(float("nan"))
    cache.v.fill_(float("nan"))
    n = rows.num_rows
    q, want, at = H.bf16(g.standard_normal((n, heads, dim))), np.zeros((n, heads, vdim)), 0
    for b, (c, x) in enumerate(entries):
        k, v = H.bf16(g.standard_normal((c + x, kv, dim))), H.bf16(g.standard_normal((c + x, kv, vdim)))
        fill(cache, table, b, t(k, torch.bfloat16), t(v, torch.bfloat16))
        for i in range(x):  # keys in the row's window
            lo = max(0, c + i - window + 1) if window else 0
            want[at + i : at + i + 1] = R.causal_attention(q[at + i : at + i + 1], k[lo : c + i + 1], v[lo : c + i + 1], dim ** -0.5, c + i - lo)
        at += x
    qd = torch.zeros(n, heads, cache.k.shape[3], device=DEV, dtype=torch.bfloat16)
    qd[..., :dim] = t(q, torch.bfloat16)
    out = torch.empty(n, heads, vdim, device=DEV, dtype=torch.bfloat16)
    ops.paged_prefill_attention(qd, cache, rows, dim ** -0.5, out, ops.AttnOptions(window=window) if window else None)
    close(out, want, torch.bfloat16)
    H.status_clear()


@pytest.mark.parametrize("heads,kv,dim,vdim", [(2, 1, 64, 48), (4, 2, 128, 128)])
@pytest.mark.parametrize("page,prior,new,window", [(16, 950, 70, 0), (16, 970, 70, 0), (16, 2041, 70, 0), (48, 1000, 133, 0), (32, 2000, 101, 0), (64, 4015, 70, 0),
                                                   (64, 4090, 70, 0), (16, 2500, 70, 1200), (32, 4500, 33, 2100), (64, 5000, 200, 4200)])
def test_prompt_attention_over_many_keys(heads, kv, dim, vdim, page, prior, new, window):
    """Keys around 1024, 2048 and 4096: the fetching warps find the places of 32 boxes of 16, 32 or 64 rows at a time, half of a
    tile's blocks each, and here need them more than once; with a window the first block is not the first.  Rows of the last page
    that no token was written to are not numbers."""
    from inference_engine_b200 import ops

    gen = torch.Generator(device=DEV).manual_seed(prior)
    rows, table, pages, _ = make_rows([(3, 1), (prior, new)], page)
    cache = ops.make_paged_kv(pages, kv, page, dim, vdim, torch.bfloat16, DEV)
    cache.k.fill_(float("nan"))
    cache.v.fill_(float("nan"))
    seqs = []
    for b, n in enumerate((4, prior + new)):
        k, v = (torch.randn(n, kv, d, generator=gen, device=DEV).to(torch.bfloat16) for d in (dim, vdim))
        p = torch.arange(n, device=DEV)
        at = torch.as_tensor(table[b], device=DEV)[p // page].long()
        cache.k[at, :, p % page], cache.v[at, :, p % page] = k, v
        seqs.append((k.double(), v.double()))
    q = torch.randn(1 + new, heads, dim, generator=gen, device=DEV).to(torch.bfloat16)
    out = ops.paged_attention(q, cache, rows, 3.0 / dim ** 0.5, ops.AttnOptions(window))
    k, v = (x.repeat_interleave(heads // kv, 1) for x in seqs[1])
    s = torch.einsum("nhd,khd->hnk", q[1:].double(), k) * (3.0 / dim ** 0.5)
    pos, key = prior + torch.arange(new, device=DEV)[:, None], torch.arange(prior + new, device=DEV)
    seen = (key <= pos) & ((key > pos - window) if window else True)
    want = torch.einsum("hnk,khd->nhd", s.masked_fill(~seen, -torch.inf).softmax(-1), v)
    close(out[1:], want.cpu().numpy(), torch.bfloat16)
    H.status_clear()


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_beyond_the_tensor_core_sizes(dtype):
    from inference_engine_b200 import ops

    g = np.random.default_rng(4)
    rows, table, pages, _ = make_rows([(37, 1), (5, 30)])
    cache = ops.make_paged_kv(pages, 1, 16, 200, 260, dtype, DEV)
    assert not ops.tensor_core_attention(cache)
    q = H.bf16(g.standard_normal((31, 2, 200)))
    want, at = np.zeros((31, 2, 260)), 0
    for b, (c, x) in enumerate([(37, 1), (5, 30)]):
        k, v = H.bf16(g.standard_normal((c + x, 1, 200))), H.bf16(g.standard_normal((c + x, 1, 260)))
        fill(cache, table, b, t(k, dtype), t(v, dtype))
        want[at : at + x] = R.causal_attention(q[at : at + x], k, v, 0.1, c)
        at += x
    close(ops.paged_attention(t(q, dtype), cache, rows, 0.1), want, dtype)


def test_decode_attention_splits_and_idle_rows():
    """Long and short entries over the whole persistent grid, entries past num_decoding, and one entry alone."""
    from inference_engine_b200 import ops

    g = np.random.default_rng(5)
    heads, kv, dim, vdim, page = 6, 3, 40, 72, 64
    for lens in ([5000, 1, 64, 65, 900, 128, 127, 2300], [3000], [70] * 40):
        B = len(lens) + 2  # two idle rows
        need = [(n + page - 1) // page for n in lens]
        table = np.full((B, max(need)), -1, np.int32)
        perm, at = g.permutation(sum(need)), 0
        for b, m in enumerate(need):
            table[b, :m] = perm[at : at + m]
            at += m
        cache = ops.make_paged_kv(sum(need), kv, page, dim, vdim, torch.bfloat16, DEV)
        cache.k[..., :dim] = torch.randn(cache.k.shape[:3] + (dim,), device=DEV)
        cache.v[..., :vdim] = torch.randn(cache.v.shape[:3] + (vdim,), device=DEV)
        rows = ops.Rows(B, i32([n - 1 for n in lens] + [7, 7]), i32([len(lens)]), i32(table))
        q = torch.randn(B, heads, dim, device=DEV).to(torch.bfloat16)
        got = ops.paged_attention(q, cache, rows, 0.3)
        again = ops.paged_attention(q, cache, rows, 0.3)
        assert torch.equal(got, again)
        assert got[len(lens) :].abs().sum().item() == 0
        kk, vv, qq = cache.k.float().cpu().numpy(), cache.v.float().cpu().numpy(), q.float().cpu().numpy()
        for b, n in enumerate(lens):
            flat = lambda x, d: np.concatenate([x[p] for p in table[b, : need[b]]], axis=1)[:, :n, :d].transpose(1, 0, 2)
            want = R.causal_attention(qq[b : b + 1], flat(kk, dim), flat(vv, vdim), 0.3, n - 1)
            close(got[b : b + 1], want, torch.bfloat16)
        close(ops.attention_rows(q, cache, rows, 0.3)[: len(lens)], got[: len(lens)].float().cpu().numpy(), torch.bfloat16)
        H.status_clear()


@pytest.mark.parametrize("heads,kv,dim,vdim,window", [(16, 8, 64, 64, 0), (16, 8, 32, 48, 200), (72, 8, 64, 24, 0)])
def test_decode_attention_of_many_narrow_heads(heads, kv, dim, vdim, window):
    """More pairs of entry and kv head than two blocks per multiprocessor, keys and values of one block of channels, with and without
    hand-offs: against the kernel for any size."""
    from inference_engine_b200 import ops

    g = np.random.default_rng(dim)
    for lens in ([1, 63, 64, 65, 130] * 8, [3000] + [200] * 37 + [1, 2]):
        B = len(lens) + 1  # one idle row
        need = [(n + 63) // 64 for n in lens]
        table = np.full((B, max(need)), -1, np.int32)
        perm, at = g.permutation(sum(need)), 0
        for b, n in enumerate(need):
            table[b, :n] = perm[at : at + n]
            at += n
        cache = ops.make_paged_kv(sum(need), kv, 64, dim, vdim, torch.bfloat16, DEV)
        cache.k[..., :dim] = torch.randn(cache.k.shape[:3] + (dim,), device=DEV)
        cache.v[..., :vdim] = torch.randn(cache.v.shape[:3] + (vdim,), device=DEV)
        rows = ops.Rows(B, i32([n - 1 for n in lens] + [7]), i32([len(lens)]), i32(table))
        q = torch.randn(B, heads, dim, device=DEV).to(torch.bfloat16)
        opt = ops.AttnOptions(window=window)
        got = ops.paged_attention(q, cache, rows, 0.3, opt)
        assert torch.equal(got, ops.paged_attention(q, cache, rows, 0.3, opt))
        close(got, ops.attention_rows(q, cache, rows, 0.3, opt).float().cpu().numpy(), torch.bfloat16)
        H.status_clear()


MOE = [  # rows, width, ff, experts, top, limit
    (1, 64, 40, 4, 1, 2.0), (37, 64, 24, 5, 3, 0.5), (5, 72, 64, 8, 8, 1.0), (700, 136, 200, 3, 2, 7.0), (300, 64, 64, 40, 6, 1.5),
    (33, 30, 18, 3, 2, 1.0), (260, 520, 96, 2, 1, 2.0),
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,width,ff,experts,top,limit", MOE)
def test_mixture(dtype, rows, width, ff, experts, top, limit):
    from inference_engine_b200 import ops

    g = np.random.default_rng(6)
    mat = lambda o, i, s: H.bf16(g.standard_normal((o, i)) * s * i ** -0.5)
    w = {"router": mat(experts, width, 2.0)}
    for e in range(experts):
        w.update({f"e{e}.gate": mat(ff, width, 3.0), f"e{e}.up": mat(ff, width, 3.0), f"e{e}.down": mat(width, ff, 1.0)})
    x = H.bf16(g.standard_normal((rows, width)))
    tt = lambda k: t(w[k], torch.bfloat16)
    ex = ops.make_experts(tt("router"), [tt(f"e{e}.gate") for e in range(experts)], [tt(f"e{e}.up") for e in range(experts)],
                          [tt(f"e{e}.down") for e in range(experts)], top, limit, 1.702, dtype, torch.device(DEV))
    want = R.mixture(np.float64(x), w, "", {"router": {"experts": experts, "top": top}, "expert": {"limit": limit}})
    ids, _ = R.route(np.float64(x), w["router"], top)
    for variant in (None, 1):
        ex.counts.zero_()
        y, places = ops.mixture(t(x), t(x, dtype), ex, variant)
        assert sorted(places.flatten().tolist()) == list(range(rows * top))
        assert ex.counts.tolist() == np.bincount(ids.flatten(), minlength=experts).tolist()
        got = y.float()[places.long()].sum(1)
        close(got, want, dtype, 1e-5 if dtype == torch.float32 else 2e-2)
    H.status_clear()


@pytest.mark.parametrize("rows,width,ff,experts,top", [(1, 2048, 512, 40, 2), (4, 2048, 1536, 40, 2), (70, 2048, 1536, 13, 4), (130, 1032, 520, 40, 3), (900, 1024, 776, 25, 5), (1000, 2048, 1280, 16, 3)])
def test_both_products_of_the_experts_in_one_launch(rows, width, ff, experts, top):
    """More items than multiprocessors, one tile alone and a few tiles of one or two rows (one row goes in two launches itself), weight blocks and
    steps with a remainder: the same bits as in two launches, again and again."""
    from inference_engine_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(rows)
    mat = lambda *s: torch.randn(*s, generator=g, device=DEV) * s[-1] ** -0.5
    ex = ops.make_experts(mat(experts, width).to(torch.bfloat16), mat(experts, ff, width), mat(experts, ff, width), mat(experts, width, ff), top, 7.0, 1.702,
                          torch.bfloat16, torch.device(DEV))
    x = torch.randn(rows, width, generator=g, device=DEV)

    def rows_of(variant):
        ex.counts.zero_()
        y, places = ops.mixture(x, x.to(torch.bfloat16), ex, variant)
        return y[places.long()]

    want = rows_of(0)
    for _ in range(5):
        assert torch.equal(rows_of(None), want)
    H.status_clear()


@pytest.mark.parametrize("rows,width,experts,top", [(600, 2052, 33, 3), (515, 4100, 5, 2), (700, 2052, 5, 2), (1190, 2052, 33, 4), (2060, 1028, 40, 2)])
def test_router_of_prompt_steps(rows, width, experts, top):
    """The router's forms for many rows: eight steps of weights in flight with a remainder behind them, few experts whose
    channels are cut into slices, and more rows than two blocks per multiprocessor hold."""
    test_mixture(torch.bfloat16, rows, width, 16, experts, top, 1.0)


def test_router_takes_rows_that_are_not_numbers():
    """Idle rows of a padded step may hold anything; they must not disturb the others or leave the expert range."""
    from inference_engine_b200 import ops

    m = H.model(H.small(), H.weights(H.small()), torch.bfloat16)
    ex = m.layers[0].experts
    x = torch.randn(9, 64, device=DEV)
    x[3] = float("nan")
    ex.counts.zero_()
    y, places = ops.mixture(x, x.to(torch.bfloat16), ex)
    assert sorted(places.flatten().tolist()) == list(range(18))
    ex.counts.zero_()
    keep = [i for i in range(9) if i != 3]
    y2, places2 = ops.mixture(x[keep].contiguous(), x[keep].to(torch.bfloat16), ex)
    assert torch.equal(y[places[keep].long()].sum(1), y2[places2.long()].sum(1))


@pytest.mark.parametrize("op", ["norm", "sum and norm", "wide norm", "rotation of many rows", "rotation of few rows", "whole norms by eights", "whole norms by pairs", "whole norms of any size"])
def test_chained_launches_wait_for_weights_and_angles(op):
    """The kernel in front writes the norm weights or the angle table of the one behind, which may be brought up meanwhile: it reads neither early."""
    from inference_engine_b200 import kernels as K
    from inference_engine_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    width = 5120 if op == "wide norm" else 2048
    front, ones = rnd(2000, width), torch.ones(width, device=DEV)
    made = front.clone()  # what the kernel in front writes, its last rows last
    n, heads, kv = 300 if "many" in op else 40, 16, 8
    dim = {"whole norms by pairs": 60, "whole norms of any size": 75}.get(op, 64)
    cache = ops.make_paged_kv(n, kv, 16, dim, dim, torch.bfloat16, DEV)
    rows = ops.Rows(n, i32(np.arange(n) % 16), i32([n]), i32(np.arange(n)[:, None]))
    qkv = rnd(n, (heads + 2 * kv) * dim).to(torch.bfloat16)
    x, delta = rnd(400, width), rnd(1600, width).to(torch.bfloat16)
    places = torch.randperm(1600, generator=g, device=DEV).int().view(400, 4)

    def behind(x):
        w = made[-1]
        if "norm" in op and "whole" not in op:
            some = "sum" in op
            return [ops.scaled_add_norm(x, delta if some else None, w, 1.5, 1e-5, torch.bfloat16, places if some else None)[1]]
        angles = made[-4:].view(-1)[: 16 * 32 * 2].view(16, 32, 2) if dim == 64 else made[-4:].view(-1)[: 16 * 20 * 2].view(16, 20, 2)
        if "whole" in op:
            q = ops.norm_rope_write(qkv, rows, cache, made[-3:].view(-1)[: heads * dim], made[-1, : kv * dim], 1e-5, angles, heads)
        else:
            q = ops.rope_write(qkv, rows, cache, angles, heads, True, True, 1e-5)
        return [q, cache.k.clone()]

    def run():
        mine = x.clone()
        made.copy_(front)
        ops.scaled_add_norm(made, None, ones, 1.0, 1e-5, torch.bfloat16)
        return behind(mine)  # nothing stands between the two

    want = run()
    K.set_early_start(True)
    try:
        for _ in range(10):
            made.fill_(float("nan"))
            for got, w in zip(run(), want):
                assert torch.equal(got, w)
    finally:
        K.set_early_start(False)
    H.status_clear()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv,dim,vdim,window", [(4, 2, 48, 40, 0), (16, 8, 112, 96, 70), (3, 3, 128, 200, 0)])
def test_attention_rows_go_by_their_own_entry_and_position(heads, kv, dim, vdim, window, dtype):
    """The entries' first rows only say how rows are shared out: positions that jump, go back or stay, idle rows, rows of other entries and rows
    behind the last entry are done as without the list.  The table has room for many more keys than there are."""
    from inference_engine_b200 import ops

    g = np.random.default_rng(dim)
    at = [(0, p) for p in [10, 11, 12, 40, 41, 7, 7, -1, *range(90, 115), 149]]
    at += [(1, p) for p in (149, 148, 147, 0, 1)] + [(0, 60), (2, 61), (2, 62), (1, 63)]
    listed = [0, 34, 34, len(at)]
    at += [(2, p) for p in (*range(20, 45), 149)] + [(0, -1), (0, 0), (1, 64)]  # of no entry in the list
    n, keys, page = len(at), 150, 16
    per = -(-keys // page)
    perm = g.permutation(3 * per + 2)
    table = np.full((3, 64), -1, np.int32)
    table[:, :per] = perm[: 3 * per].reshape(3, per)
    cache = ops.make_paged_kv(3 * per + 2, kv, page, dim, vdim, dtype, DEV)
    k, v = H.bf16(g.standard_normal((3, keys, kv, dim))), H.bf16(g.standard_normal((3, keys, kv, vdim)))
    for b in range(3):
        fill(cache, table, b, t(k[b], dtype), t(v[b], dtype))
    q, want = H.bf16(g.standard_normal((n, heads, dim))), np.zeros((n, heads, vdim))
    for r, (b, p) in enumerate(at):
        lo = max(0, p - window + 1) if window else 0
        if p >= 0:
            want[r : r + 1] = R.causal_attention(q[r : r + 1], k[b, lo : p + 1], v[b, lo : p + 1], dim ** -0.5, p - lo)
    qd = torch.zeros(n, heads, cache.k.shape[3], device=DEV, dtype=dtype)
    qd[..., :dim] = t(q, dtype)
    for cu in (None, i32(listed), torch.tensor(listed, device=DEV), i32([0] * 40 + [n]), i32([0, n])):
        rows = ops.Rows(n, i32([0] * 3), i32([0]), i32(table), i32([b for b, _ in at]), i32([p for _, p in at]), cu)
        out = torch.full((n, heads, vdim), float("nan"), device=DEV, dtype=dtype)
        ops.attention_rows(qd, cache, rows, dim ** -0.5, ops.AttnOptions(window=window), out)
        close(out, want, dtype)
    H.status_clear()
