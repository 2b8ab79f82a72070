"""Operands that the previous call on the stream has just written, where that call announces itself early: a Linear's bias, a norm's
scale.  Only a Linear's weight may be read ahead of the stream order.

The same calls with a synchronisation between them give the reference, so both sides are equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(xn, first, second):
    torch.cuda.synchronize()
    v = first()
    torch.cuda.synchronize()
    want = second(v)
    torch.cuda.synchronize()
    v.zero_()
    torch.cuda.synchronize()
    got = second(first())
    torch.cuda.synchronize()
    return got, want


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 9, 40, 100, 300])
@pytest.mark.parametrize("n", [640, 4096])
def test_bias(xn, cuda, dtype, rows, n):
    g = torch.Generator(device=cuda).manual_seed(n + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda).to(dtype)
    cond, w = xn.Linear(rnd(n, 4096)), rnd(n, 1024)
    x = rnd(rows, 1024)
    for _ in range(5):
        c = rnd(1, 4096)
        got, want = _chain(xn, lambda: cond(c), lambda v: xn.Linear(w, v.view(n))(x))
        assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 16, 2000])
@pytest.mark.parametrize("cols", [512, 4096])
def test_norm_scale(xn, cuda, dtype, rows, cols):
    g = torch.Generator(device=cuda).manual_seed(cols + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda).to(dtype)
    cond, x = xn.Linear(rnd(cols, 4096)), rnd(rows, cols)
    for _ in range(5):
        c = rnd(1, 4096)
        got, want = _chain(xn, lambda: cond(c), lambda v: xn.ops.rms_norm(x, v.view(cols), 1e-5))
        assert torch.equal(got, want)
