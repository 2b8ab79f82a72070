"""The tiled tensor-memory kernel with the tiles of its last, partly filled round cut along k: few tiles and many, ragged
rows, columns and k, two row blocks per tile, both fp8 variants, a bias, batches, and a captured launch.

Bounds: as in test_few_rows_gpu.py, |y - ref| <= u |ref| + k 2^-23 sum|a||b| (the tensor cores add with truncation: one
ulp per step instead of half) with one more u where a bias is added to the rounded product."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _check(y, a, b, u, bias=None):
    a64, b64 = a.double(), b.double().transpose(-1, -2)
    ref, mag = a64 @ b64, a64.abs() @ b64.abs()
    lim = u * ref.abs() + a.shape[-1] * 2.0 ** -23 * mag
    if bias is not None:
        ref = ref + bias.double()
        lim = lim + u * ref.abs()
    err = (y.double() - ref).abs()
    assert not torch.isnan(y).any()
    assert bool((err <= lim).all()), float((err / lim).max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,bias", [(1024, 5120, 4168, False), (1000, 5001, 2048, True), (520, 3000, 11264, False),
                                        (3001, 4096, 2056, True), (1300, 8200, 1024, False), (257, 4096, 4096, True)])
def test_16bit(xn, cuda, dtype, m, n, k, bias):
    g = torch.Generator(device=cuda).manual_seed(m + n)
    x = torch.randn(m, k, generator=g, device=cuda).to(dtype)
    w = (torch.randn(n, k, generator=g, device=cuda) * 0.02).to(dtype)
    b = torch.randn(n, generator=g, device=cuda).to(dtype) if bias else None
    layer = xn.Linear(w, b)
    y = layer(x)
    _check(y, x, w, U[dtype], b)
    for _ in range(3):  # the sums run in a fixed order
        assert torch.equal(layer(x), y)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("m,n,k", [(1024, 5120, 4096), (300, 7000, 4112), (4096, 4096, 2048)])
def test_e4m3(xn, cuda, variant, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(n)
    x = torch.randn(m, k, generator=g, device=cuda).to(torch.bfloat16)
    wq, ws = xn.quantize_weights_fp8(torch.randn(n, k, generator=g, device=cuda) * 0.02)
    hi, lo, xs = xn.split_rows_e4m3(x, True)
    e = lambda t: t.view(torch.float8_e4m3fn).double()
    a = (e(hi) + (e(lo) if variant == 0 else 0.0)) * xs.double()[:, None]
    y = xn.linear_fp8(x, wq, ws, variant)
    _check(y, a, e(wq) * ws.double()[:, None], U[torch.bfloat16])
    assert torch.equal(xn.linear_fp8(x, wq, ws, variant), y)


def test_batches_and_a_row_major_right_hand_side(xn, cuda):
    g = torch.Generator(device=cuda).manual_seed(3)
    x = torch.randn(3, 700, 2048, generator=g, device=cuda).to(torch.bfloat16)
    w = torch.randn(3, 2200, 2048, generator=g, device=cuda).to(torch.bfloat16)
    _check(xn.matmul_t(x, w), x, w, U[torch.bfloat16])
    _check(xn.matmul(x, w.transpose(1, 2).contiguous()), x, w, U[torch.bfloat16])


def test_captured(xn, cuda):
    g = torch.Generator(device=cuda).manual_seed(4)
    x = torch.randn(1024, 4096, generator=g, device=cuda).to(torch.bfloat16)
    w = torch.randn(5120, 4096, generator=g, device=cuda).to(torch.bfloat16)
    layer = xn.Linear(w)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        layer(x)
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        y = layer(x)
    graph.replay()
    torch.cuda.synchronize()
    _check(y, x, w, U[torch.bfloat16])
