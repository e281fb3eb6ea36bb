"""apus_cuda_sparse_attn_batch_dev takes any stream and returns before the work is done: what it keeps between its
kernels (scores, compacted ids, walk flags) belongs to the one call.  Two calls of different sizes and values run
side by side on two streams, from two threads on one stream, and out of one graph beside another; every result is
the bits of the same call alone."""
import threading

import numpy as np
import pytest

from _gpu import lib
from apus_b200 import check

pytestmark = pytest.mark.gpu
H, D = 64, 512


class Call:
    """One decode step's attention over the caller's BF16 rows; `wild` rows hold values outside the window in which
    a product of two BF16 values is exact, so that the call needs the two-instruction walk."""

    def __init__(self, seed, B, n, wild):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed)
        rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
        self.B, self.n = B, n
        self.q, self.sink = rnd(B, H, D).bfloat16().float(), rnd(H)
        self.kv = rnd(B, n + 7, D).bfloat16()
        if wild:
            self.kv[:, :, 3] *= 2.0 ** -70
            self.q[:, :, 5] *= 1.0009765625 + 2.0 ** -20
        self.idx = torch.stack([torch.randperm(n + 7, generator=g, device="cuda")[:n] for _ in range(B)]).int()
        self.idx[:, ::5] = -1                                      # dropped, the order of the rest is kept
        self.o = torch.empty(B, H, D, device="cuda")
        torch.cuda.synchronize()

    def run(self, stream):
        check(lib().apus_cuda_sparse_attn_batch_dev(self.q.data_ptr(), self.sink.data_ptr(), H, D, self.idx.data_ptr(), self.n, self.B,
                                                    D ** -0.5, self.kv.data_ptr(), 0, 0, self.kv.data_ptr(), self.n + 7, self.n + 7,
                                                    self.o.data_ptr(), stream.cuda_stream))

    def bits(self):
        return self.o.cpu().numpy().view(np.uint32).copy()


@pytest.fixture
def pair():
    import torch
    a, b = Call(1, 3, 640, False), Call(2, 5, 333, True)
    s = torch.cuda.Stream(), torch.cuda.Stream()
    want = []
    for c in (a, b):
        c.run(s[0])
        torch.cuda.synchronize()
        want.append(c.bits())
        c.o.fill_(float("nan"))
    torch.cuda.synchronize()
    return a, b, s, want


def same(pair):
    import torch
    torch.cuda.synchronize()
    a, b, _, want = pair
    assert np.array_equal(a.bits(), want[0]) and np.array_equal(b.bits(), want[1])


def test_two_streams(pair):
    a, b, s, _ = pair
    for _ in range(20):
        a.run(s[0])
        b.run(s[1])
    same(pair)


def test_two_threads_on_one_stream_with_growing_sizes(pair):
    a, b, s, _ = pair
    big = [Call(10 + k, 2 * k + 1, 700, False) for k in range(4)]
    errs = []

    def work(calls):
        try:
            for c in calls * 10:
                c.run(s[0])
        except Exception as e:                                     # noqa: BLE001 -- shown by the main thread
            errs.append(e)
    t = [threading.Thread(target=work, args=(c,)) for c in ([a], [b, *big])]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not errs, errs
    same(pair)


def test_recorded_beside_a_call(pair):
    """Recorded on a stream that has never run the call; replayed while the other call runs, also after calls that
    needed more scratch."""
    import torch
    a, b, s, _ = pair
    graph, rec = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=rec):
        a.run(rec)
    Call(30, 9, 1000, False).run(s[1])
    for _ in range(20):
        with torch.cuda.stream(s[0]):
            graph.replay()
        b.run(s[1])
    same(pair)
    del graph


def test_more_streams_than_buffers_are_kept(pair):
    import torch
    a, b, s, _ = pair
    streams = [torch.cuda.Stream() for _ in range(20)]
    for k in range(3):
        for t in streams:
            b.run(s[1])
            a.run(t)
    same(pair)
