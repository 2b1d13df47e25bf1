"""Decode attention behind the launcher boundary (csrc/attention.cu): slices and their merge meet in memory of the call, whatever else runs at the same time."""
import threading

import pytest

torch = pytest.importorskip("torch")
from ntransformer_b200 import kernels as K  # noqa: E402
from ntransformer_b200._lib import lib  # noqa: E402

pytestmark = [pytest.mark.gpu]


class Call:
    def __init__(self, seed, heads, kv, dim, ctx):
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.shape = (ctx, heads, kv, dim)
        self.q = torch.randn(heads, dim, device="cuda", generator=g)
        self.kc, self.vc = (torch.randn(ctx, kv, dim, device="cuda", generator=g).half() for _ in range(2))
        self.alone = self(torch.empty_like(self.q))
        torch.cuda.synchronize()

    def __call__(self, out, stream=None):
        ctx, heads, kv, dim = self.shape
        K.launch_attention_decode(out, self.q, self.kc, self.vc, ctx, heads, kv, dim, ctx, dim ** -0.5, stream)
        return out


CALLS = [(1, 64, 8, 128, 4000), (2, 32, 8, 128, 900), (3, 16, 2, 64, 2500), (4, 64, 8, 128, 70)]


def test_alone():
    for c in map(lambda a: Call(*a), CALLS):
        ctx, heads, kv, dim = c.shape
        k, v = (t.double().repeat_interleave(heads // kv, 1) for t in (c.kc, c.vc))
        w = torch.softmax(torch.einsum("hd,shd->hs", c.q.double(), k) * dim ** -0.5, 1)
        want = torch.einsum("hs,shd->hd", w, v)
        assert ((c.alone - want).norm() / want.norm()).item() <= 5e-6


def test_several_streams_at_once():
    calls, streams = [Call(*a) for a in CALLS], [torch.cuda.Stream() for _ in CALLS]
    outs = [[torch.full_like(c.q, 7.0) for _ in range(50)] for c in calls]
    torch.cuda.synchronize()
    for i in range(50):
        for c, s, o in zip(calls, streams, outs):
            c(o[i], s)
    torch.cuda.synchronize()
    assert all(torch.equal(x, c.alone) for c, o in zip(calls, outs) for x in o)


def test_several_threads_on_one_stream_and_on_their_own():
    calls, shared = [Call(*a) for a in CALLS], torch.cuda.Stream()
    outs = [[torch.full_like(c.q, 7.0) for _ in range(100)] for c in calls]
    torch.cuda.synchronize()

    def work(c, o, own):
        for i, x in enumerate(o):
            c(x, own if i % 2 else shared)

    threads = [threading.Thread(target=work, args=(c, o, torch.cuda.Stream())) for c, o in zip(calls, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert all(torch.equal(x, c.alone) for c, o in zip(calls, outs) for x in o)
    lib().nt_b200_trim_memory()
    x = calls[0](torch.empty_like(calls[0].q))
    torch.cuda.synchronize()
    assert torch.equal(x, calls[0].alone)


def test_captured():
    a, b = Call(*CALLS[0]), Call(*CALLS[1])
    outs = [torch.full_like(c.q, 7.0) for c in (a, b, a)]
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        for c, o in zip((a, b, a), outs):
            c(o)
            o += 0                                                # a launch that is not this library's between two of its
    for _ in range(3):
        for o in outs:
            o.fill_(7.0)
        graph.replay()
        b(torch.empty_like(b.q))                                  # and one on another stream beside it
        torch.cuda.synchronize()
        assert all(torch.equal(o, c.alone) for c, o in zip((a, b, a), outs))
