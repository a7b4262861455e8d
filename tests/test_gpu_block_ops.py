"""GPU parity of the decoder block's element-wise ops (silu_mul, add_rms_norm) against the reference kernels'
own outputs (golden) and against the CPU oracle on other shapes.  The residual stream must be exact; the
normalised / activated outputs may differ by one bf16 step where exp / rsqrt differ in their last place."""
import os

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests import helpers as H
from tests.test_oracle_block_ops import GOLD, ulps

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from inference_engine_b200 import kernels

    return kernels


def close(got_bits, want_bits, frac=0.01):
    d = ulps(got_bits, want_bits)
    assert d.max() <= 1 and (d > 0).mean() < frac, (int(d.max()), float((d > 0).mean()))


def test_reference_golden(K):
    g = dict(np.load(GOLD))
    y = K.silu_mul(H.bits_tensor(g["sm_in_bf16"]))
    close(H.to_bits(y), g["sm_out_bf16"])
    r, n = K.add_rms_norm(H.bits_tensor(g["arn_res_bf16"]), H.bits_tensor(g["arn_delta_bf16"]),
                          H.bits_tensor(g["arn_w_bf16"]), 1e-6)
    assert np.array_equal(H.to_bits(r), g["arn_new_res_bf16"])
    close(H.to_bits(n), g["arn_normed_bf16"])


@pytest.mark.parametrize("N,D", [(1, 8), (3, 2048), (33, 6144), (1024, 2048), (2, 8192)])
def test_add_rms_norm_vs_oracle(K, N, D):
    rng = np.random.default_rng(N * 7 + D)
    res, delta = H.randn_bf16(rng, N, D) * 4, H.randn_bf16(rng, N, D)
    res = O.bf16_round(res)
    w = O.bf16_round((1 + 0.1 * rng.standard_normal(D)).astype(np.float32))
    want_r, want_n = O.add_rms_norm(res, delta, w, 1e-6)
    r, n = K.add_rms_norm(H.bf16_tensor(res), H.bf16_tensor(delta), H.bf16_tensor(w), 1e-6)
    assert np.array_equal(H.to_bits(r), O.bf16_bits(want_r))
    close(H.to_bits(n), O.bf16_bits(want_n))


@pytest.mark.parametrize("N,D", [(1, 8), (5, 1536), (64, 6144), (7, 12288)])
def test_silu_mul_vs_oracle_strided(K, N, D):
    rng = np.random.default_rng(N + D)
    buf = O.bf16_round(H.randn_bf16(rng, N, 2 * D + 64) * 3)
    t = H.bf16_tensor(buf)[:, : 2 * D]  # a strided view, like a slice of a wider projection
    y = K.silu_mul(t)
    close(H.to_bits(y), O.bf16_bits(O.silu_mul(buf[:, : 2 * D])))


def test_argument_checks(K):
    x = torch.zeros(4, 2 * 12, dtype=torch.bfloat16, device="cuda")  # D = 12: not a multiple of 8
    with pytest.raises(ValueError):
        K.silu_mul(x)
    big = torch.zeros(2, 8200, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ValueError):
        K.add_rms_norm(big, big, torch.ones(8200, dtype=torch.bfloat16, device="cuda"), 1e-6)


@pytest.mark.parametrize("chained", [False, True])
def test_branches_of_a_recorded_graph(K, chained):
    """Calls side by side, one branch cut into two and one left empty: each starts behind what came before, what follows waits for all."""
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(3, 512, 4096, generator=g, device="cuda").to(torch.bfloat16)
    from inference_engine_b200 import _lib

    lib = _lib.load()

    def call():
        first = K.silu_mul(x[0])
        with K.Branches(lib) as b:
            kept = [torch.cat([first, first], dim=1)]  # what a branch allocates lives until the end
            a = K.silu_mul(kept[0])
            with K.Branches(lib) as c:
                d = K.silu_mul(x[1])
                c.next()
                e = K.silu_mul(x[2])
                c.next()
            kept.append(torch.cat([d, e], dim=1))
            f = K.silu_mul(kept[1])
            b.next()
            kept += [first + 1]
            kept += [torch.cat([first, kept[2]], dim=1)]
            h = K.silu_mul(kept[3])
        return K.silu_mul(torch.cat([a + f, h], dim=1)), first

    want = call()
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    K.set_early_start(chained)
    try:
        with torch.cuda.graph(graph, stream=s):
            got = call()
    finally:
        K.set_early_start(False)
    for _ in range(3):
        graph.replay()
        assert all(torch.equal(u, v) for u, v in zip(want, got))
    x.mul_(0.5)
    want = call()
    graph.replay()
    assert all(torch.equal(u, v) for u, v in zip(want, got))


def test_branches_at_the_start_of_a_graph(K):
    """Nothing stands in front of the fork, and the last branch is empty."""
    from inference_engine_b200 import _lib

    x = torch.randn(2, 64, 256, device="cuda").to(torch.bfloat16)
    K.silu_mul(x[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with K.Branches(_lib.load()) as b:
            a = K.silu_mul(x[0])
            b.next()
            c = K.silu_mul(x[1])
            b.next()
        d = K.silu_mul(torch.cat([a, c], dim=1))
    graph.replay()
    assert torch.equal(d, K.silu_mul(torch.cat([K.silu_mul(x[0]), K.silu_mul(x[1])], dim=1)))


def edges_of(body, *streams):
    """What `body` records on each of the streams: (edges, chained ones among them)."""
    import ctypes

    from cuda.bindings import runtime as rt

    driver = ctypes.CDLL("libcuda.so.1")

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r
        return r[1:]

    for s in streams:
        ok(rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed))
    try:
        body()
    finally:
        graphs = [rt.cudaStreamEndCapture(s.cuda_stream) for s in streams]
    out = []
    for r in graphs:
        (g,) = ok(r)
        count = ctypes.c_size_t(64)
        ends, data = (ctypes.c_void_p * 64)(), (ctypes.c_uint8 * 8 * 64)()  # data: from port, to port, type, reserved
        assert driver.cuGraphGetEdges_v2(ctypes.c_void_p(int(g)), ends, (ctypes.c_void_p * 64)(), data, ctypes.byref(count)) == 0
        out.append((count.value, sum(d[2] == 1 for d in data[: count.value])))
        ok(rt.cudaGraphDestroy(g))
    return out


def test_first_launches_of_branches_and_behind_them_are_plain_on_their_stream_alone(K):
    """Chained launches: neither launches on another stream in between nor branches of the other library change which ones are plain."""
    from inference_engine_b200 import _lib

    lib, dec = _lib.load(), _lib.load_decoder()
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    x, y = (torch.zeros(4, n, dtype=torch.bfloat16, device="cuda") for n in (128, 64))
    silu = lambda on: _lib.check(lib.b200kv_silu_mul(x.data_ptr(), 128, y.data_ptr(), 64, 4, 64, on.cuda_stream), "silu_mul")
    silu_dec = lambda on: _lib.check(dec.b200dec_silu_mul(x.data_ptr(), 128, 2, y.data_ptr(), 64, 4, 64, on.cuda_stream), "silu_mul")

    def elsewhere():
        silu(s)
        b = lib.b200kv_branches_begin(s.cuda_stream)
        silu(other)
        silu(s)
        assert lib.b200kv_branches_next(b) == 0
        silu(other)
        silu(s)
        assert lib.b200kv_branches_end(b) == 0
        silu(other)
        silu(s)
        silu(s)

    def two_libraries():
        silu_dec(s)
        with torch.cuda.stream(s), K.Branches(lib) as b:
            silu_dec(s)  # the first of its branch, though of the other library
            b.next()
            silu(s)
        silu(s)  # behind the join: plain; from here on nothing is
        silu_dec(s)
        silu(s)

    silu(s), silu_dec(s), torch.cuda.synchronize()
    K.set_early_start(True)
    try:
        # 0 -> 1, 0 -> 2, 1 -> 3, 2 -> 3 plain, 3 -> 4 chained; the other stream's three launches a chain
        assert edges_of(elsewhere, s, other) == [(5, 1), (2, 2)]
        # 0 -> 1, 0 -> 2, 1 -> 3, 2 -> 3 plain, 3 -> 4 -> 5 chained
        assert edges_of(two_libraries, s) == [(6, 2)]
    finally:
        K.set_early_start(False)
