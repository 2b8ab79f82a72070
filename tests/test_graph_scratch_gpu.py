"""Captured calls that hand data over through scratch have a block of their graph's own: they run as they do eagerly (equal bits), need no
call before them, may be replayed beside anything, and give the block back with the graph."""
import gc
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _calls(xn, device):
    g = torch.Generator(device=device).manual_seed(7)
    rnd = lambda *s, dtype=torch.bfloat16: torch.randn(*s, generator=g, device=device).to(dtype)
    out = []
    for m, n, k in ((200, 1024, 11264), (300, 2048, 8192), (1024, 5120, 4096)):  # cut tiles: few and all, few and some
        layer, x = xn.Linear(rnd(n, k), rnd(n)), rnd(m, k)
        out.append(lambda layer=layer, x=x: layer(x))
    fp8, x8 = xn.LinearFp8.from_weight(rnd(1024, 8192, dtype=torch.float32)), rnd(256, 8192)
    out.append(lambda: fp8(x8))
    a, b = rnd(3, 70, 1501), rnd(3, 1501, 256)  # rows off 16-byte boundaries
    out.append(lambda: xn.matmul(a, b))
    return out


def _capture(calls, stream=None):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = [f() for f in calls]
    return graph, y


def test_cold_captures_equal_eager_calls(xn, cuda):
    calls = _calls(xn, cuda)
    want = [f() for f in calls]  # loads the kernels
    torch.cuda.synchronize()
    xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
    graph, y = _capture(calls)
    for _ in range(3):
        for t in y:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(y, want):
            assert torch.equal(a, b)


def test_replays_beside_eager_calls_and_another_graph(xn, cuda):
    calls = _calls(xn, cuda)
    want = [f() for f in calls]
    torch.cuda.synchronize()
    g1, y1 = _capture(calls)
    g2, y2 = _capture(calls[::-1])
    s1, s2, s3 = (torch.cuda.Stream() for _ in range(3))
    for _ in range(10):
        with torch.cuda.stream(s1):
            g1.replay()
        with torch.cuda.stream(s2):
            g2.replay()
        with torch.cuda.stream(s3):
            y3 = [f() for f in calls]
        torch.cuda.synchronize()
        for a, b, c, d in zip(y1, y2[::-1], y3, want):
            assert torch.equal(a, d) and torch.equal(b, d) and torch.equal(c, d)


def test_blocks_come_back_with_their_graph(xn, cuda):
    calls = _calls(xn, cuda)[:1]
    calls[0]()
    torch.cuda.synchronize()
    xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
    pool = torch.cuda.graph_pool_handle()

    def run():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, pool=pool):
            calls[0]()
        graph.replay()
        torch.cuda.synchronize()
        graph.reset()

    def settle():  # the driver lets go of a graph's objects on a thread of its own
        gc.collect()
        torch.cuda.synchronize()
        time.sleep(0.3)

    run()
    settle()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(20):
        run()
        settle() if _ % 5 == 0 else None
    settle()
    assert free0 - torch.cuda.mem_get_info()[0] < 64 << 20
    xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
    assert torch.cuda.mem_get_info()[0] >= free0
