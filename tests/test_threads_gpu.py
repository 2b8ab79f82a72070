"""Several host threads on ONE stream: the launches of a call that hands data over through the stream's scratch (tiles cut along k,
repacked f32 operands, re-pitched rows, unpacked block weights) stay together, so every thread gets the results it gets alone.

The kernels add in a fixed order: results are equal, not merely close."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _calls(xn, device):
    g = torch.Generator(device=device).manual_seed(11)
    rnd = lambda *s, dtype=torch.bfloat16: torch.randn(*s, generator=g, device=device).to(dtype)
    prompts = []
    for m, n, k in ((3001, 4096, 2056), (1500, 4096, 2056), (300, 2048, 8192), (257, 4096, 4096)):  # cut tiles of different counts
        layer, x = xn.Linear(rnd(n, k), rnd(n)), rnd(m, k)
        prompts.append(lambda layer=layer, x=x: layer(x))
    fp8, x8 = xn.LinearFp8.from_weight(rnd(4096, 4096, dtype=torch.float32)), rnd(300, 4096)
    odd_x, odd_w = rnd(3, 70, 1501), rnd(3, 1501, 256)
    odd_x2, odd_w2 = rnd(1, 65, 1003), rnd(1, 1003, 384)
    f_x, f_w = rnd(200, 1024, dtype=torch.float32), rnd(512, 1024, dtype=torch.float32)
    f_x2, f_w2 = rnd(130, 2048, dtype=torch.float32), rnd(300, 2048, dtype=torch.float32)
    q4, xq = xn.LinearQ4.from_weight(rnd(1024, 1024, dtype=torch.float32)), rnd(200, 1024, dtype=torch.float32)
    return [[prompts[0], lambda: fp8(x8), lambda: xn.matmul(odd_x, odd_w), lambda: xn.matmul_t(f_x, f_w)],
            [prompts[1], prompts[2], lambda: xn.matmul(odd_x2, odd_w2), lambda: q4(xq)],
            [prompts[3], prompts[0], lambda: xn.matmul_t(f_x2, f_w2), lambda: q4(xq)]]


def test_threads_on_one_stream(xn, cuda):
    work = _calls(xn, cuda)
    want = [[f() for f in w] for w in work]
    torch.cuda.synchronize()
    wrong, failed = [], []
    start = threading.Barrier(len(work))

    def run(i):
        try:
            torch.cuda.set_device(cuda)
            start.wait()
            for rep in range(40):
                for j, f in enumerate(work[i]):
                    y = f()
                    if rep % 4 == 3 and not torch.equal(y, want[i][j]):
                        wrong.append((i, j, rep))
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    assert not wrong, wrong


def test_scratch_released_while_another_thread_calls(xn, cuda):
    """No block is freed between a call's scratch lookup and its last launch."""
    work = [f for w in _calls(xn, cuda) for f in w]
    want = [f() for f in work]
    torch.cuda.synchronize()
    stop, failed = threading.Event(), []

    def release():
        try:
            torch.cuda.set_device(cuda)
            while not stop.is_set():
                xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    t = threading.Thread(target=release)
    t.start()
    try:
        for _ in range(10):
            for f, w in zip(work, want):
                assert torch.equal(f(), w)
    finally:
        stop.set()
        t.join()
    assert not failed, failed
