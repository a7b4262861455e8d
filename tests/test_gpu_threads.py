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


@pytest.mark.parametrize("makers", [(attention_rows(16), attention_rows(128))], ids=["attention_rows"])
def test_sizes_side_by_side(makers, monkeypatch):
    side_by_side(monkeypatch, makers)
