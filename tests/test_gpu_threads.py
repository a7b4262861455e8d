"""Host threads that launch one kernel for different sizes, each on a stream of its own: what a call sets up for its launch
is not taken from it by another thread's call.  The threads make the library calls that the ops make, over and over, so that they
are inside the library at the same time."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


class Recorded:
    """The library, which notes the last call that is made through it."""

    def __init__(self, lib):
        self.lib = lib

    def __getattr__(self, name):
        fn = getattr(self.lib, name)

        def call(*args):
            self.last = fn, args
            return fn(*args)

        return call


def side_by_side(monkeypatch, makers, times=20000):
    from inference_engine_b200 import ops

    lib = Recorded(ops._lib_dec())
    monkeypatch.setattr(ops, "_lib_dec", lambda: lib)
    work = []
    for make in makers:
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            call = make()
            kept, out = call()
        stream.synchronize()
        work.append((lib.last, stream, kept, out, out.clone()))
    start, codes = threading.Barrier(len(work)), []

    def repeat(fn, args):
        torch.cuda.synchronize()  # the thread has a context
        start.wait()
        codes.append({fn(*args) for _ in range(times)})

    threads = [threading.Thread(target=repeat, args=w[0]) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [{0}] * len(work)
    for _, _, _, out, alone in work:
        assert torch.equal(out, alone)


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def attention_rows(dim):
    from inference_engine_b200 import ops

    def make():
        cache = ops.make_paged_kv(4, 2, 16, dim, dim, torch.float32, DEV)
        cache.k.normal_()
        cache.v.normal_()
        q = torch.randn(3, 4, dim, device=DEV)
        rows = ops.Rows(3, i32([20, 7, 15]), i32([3]), i32([[0, 1], [2, -1], [3, -1]]))

        def call():
            out = ops.attention_rows(q, cache, rows, dim ** -0.5)
            return (cache, q, rows), out

        return call

    return make


def router(rows, width):
    from inference_engine_b200 import kernels as K
    from inference_engine_b200 import ops

    def make():
        x, w = torch.randn(rows, width, device=DEV), torch.randn(5, width, device=DEV, dtype=torch.bfloat16)
        ids, ranks, counts = (torch.zeros(n, dtype=torch.int32, device=DEV) for n in (2 * rows, 2 * rows, 5))
        scores = torch.zeros(2 * rows, device=DEV)

        def call():
            args = [t.data_ptr() for t in (ids, scores, ranks, counts)]
            assert ops._lib_dec().b200dec_router(x.data_ptr(), w.data_ptr(), rows, width, 5, 2, *args, K._stream()) == 0
            return (x, w, ids, ranks, counts), scores

        return call

    return make


def norm(width):
    from inference_engine_b200 import ops

    def make():
        x, w = torch.randn(2, width, device=DEV), torch.rand(width, device=DEV)

        def call():
            return (x, w), ops.scaled_add_norm(x, None, w, 1.0, 1e-6, torch.bfloat16, keep=False)[1]

        return call

    return make


def decode_attention(entries):
    from inference_engine_b200 import ops

    def make():
        cache = ops.make_paged_kv(4, 2, 16, 64, 64, torch.bfloat16, DEV)
        cache.k.normal_()
        cache.v.normal_()
        q = torch.randn(entries, 4, 64, device=DEV).to(torch.bfloat16)
        rows = ops.Rows(entries, i32([15] * entries), i32([entries]), i32([[e % 4] for e in range(entries)]))

        def call():
            return (cache, q, rows), ops.paged_attention(q, cache, rows, 0.125)

        return call

    return make


def recurrent_step(dim, vdim, variant):
    """No entry decodes, so that the states stay as they are."""
    from inference_engine_b200 import ops

    def make():
        rec = ops.Recurrence(2, 1, dim, vdim, torch.randn(4, 2 * dim + 2 * vdim, device=DEV), None, -torch.ones(2, device=DEV),
                             torch.zeros(2, device=DEV), torch.ones(2, device=DEV), 2 * vdim + dim, 2 * vdim, 0)
        st = ops.make_recurrent_state(rec, 1, torch.bfloat16, DEV)
        x, step = torch.randn(1, rec.channels, device=DEV).to(torch.bfloat16), torch.randn(1, 2, device=DEV).to(torch.bfloat16)
        rows = ops.Rows(1, i32([3]), i32([0]), i32([[0]]), slots=i32([0]))
        out = torch.zeros(1, 2 * vdim, device=DEV)

        def call():
            ops.recurrence_decode(rec, st, x, step, None, rows, out, variant=variant)
            return (rec, st, x, step, rows), out

        return call

    return make


PAIRS = {
    "attention_rows": (attention_rows(16), attention_rows(128)),
    "router": (router(3, 64), router(3, 20000)),
    "router_of_many_rows": (router(600, 64), router(600, 4096)),
    "norm_of_any_width": (norm(33), norm(45001)),
    "decode_attention": (decode_attention(1), decode_attention(1500)),
    "recurrent_step": (recurrent_step(48, 64, 0), recurrent_step(64, 64, 0)),
    "recurrent_step_of_any_size": (recurrent_step(8, 8, 1), recurrent_step(4000, 8, 1)),
}


@pytest.mark.parametrize("name", PAIRS)
def test_sizes_side_by_side(name, monkeypatch):
    side_by_side(monkeypatch, PAIRS[name])
