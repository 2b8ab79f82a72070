"""Both sides of the lines between the kernels for 1 to 128 rows: the size just below a line and the size on it, ragged where the line allows.

Bound: one rounding to the element type of an f32 sum of exact products; tcgen05 adds with truncation, so a sum over k elements
carries at most (k / 16) 2^-23 of sum|a||b| beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (66, 4096, 504), (66, 4096, 512), (80, 4104, 1016), (80, 4104, 1024), (96, 8200, 1472), (96, 8200, 1480), (128, 4096, 1016),
    (128, 4096, 1024), (128, 4100, 2616), (128, 4100, 2624), (128, 9472, 4096), (128, 9472, 4104), (94, 4608, 1408),  # cluster / tiled
    (12, 2048, 1024), (12, 2056, 1024), (16, 2056, 2040), (16, 2056, 2048)])                                        # streaming / cluster
def test_16bit(xn, cuda, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device=cuda).bfloat16()
    w = (torch.randn(n, k, generator=g, device=cuda) * 0.05).bfloat16()
    ref, mag = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    bound = 2.0 ** -8 * ref.abs() + k / 16 * 2.0 ** -23 * mag
    assert bool(((xn.Linear(w)(x).double() - ref).abs() <= bound).all())
    if n % 8 == 0:
        assert bool(((xn.matmul(x, w.t().contiguous()).double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("variant,m,n,k", [
    (1, 8, 12288, 4096), (1, 8, 4096, 4096), (1, 8, 4096, 4112), (1, 1, 20464, 4096), (1, 1, 20480, 4096), (0, 1, 3056, 4096),
    (0, 1, 3072, 4096),                                                                                             # streaming / cluster
    (0, 128, 4096, 1024), (0, 128, 4096, 1040), (1, 128, 4096, 2032), (1, 128, 4096, 2048), (0, 96, 8200, 1472), (0, 96, 8200, 1488),
    (1, 96, 8200, 2944), (1, 96, 8200, 2960)])                                                                      # cluster / tiled
def test_e4m3(xn, cuda, variant, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device=cuda).bfloat16()
    wq, ws = xn.quantize_weights_fp8(torch.randn(n, k, generator=g, device=cuda) * 0.02)
    hi, lo, xs = xn.split_rows_e4m3(x)
    f = lambda t: t.view(torch.float8_e4m3fn).double()
    a = (f(hi) + (f(lo) if variant == 0 else 0.0)) * xs.double()[:, None]
    w = f(wq) * ws.double()[:, None]
    ref, mag = a @ w.t(), (a.abs() + (f(lo).abs() * xs.double()[:, None] if variant == 0 else 0.0)) @ w.abs().t()
    bound = 2.0 ** -8 * ref.abs() + k / 32 * 2.0 ** -22 * mag
    assert bool(((xn.linear_fp8(x, wq, ws, variant).double() - ref).abs() <= bound).all())
