"""The tensor-memory kernel for up to 128 rows: every cluster size, ragged channels and rows, k that is no multiple of a
stage, both weight layouts, nn::Linear's bias.

Bound: one rounding to the element type of an f32 sum of exact products; tcgen05 adds with truncation, so a sum over k
elements carries at most (k / 16) 2^-23 of sum|a||b| beside it; the bias is a second rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu
U = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,bias", [(17, 128, 64, False), (20, 1000, 1032, True), (64, 4100, 2048, True), (33, 257, 8192, False),
                                        (48, 20000, 512, False), (65, 300, 4096, True), (128, 1024, 1024, False), (16, 512, 11264, True),
                                        (8, 300, 12288, True), (1, 4096, 8200, True)])
def test_16bit_rows(xn, cuda, dtype, m, n, k, bias):
    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device=cuda).to(dtype)
    w = (torch.randn(n, k, generator=g, device=cuda) * 0.05).to(dtype)
    b = torch.randn(n, generator=g, device=cuda).to(dtype) if bias else None
    x64, w64 = x.double(), w.double()
    ref, mag = x64 @ w64.t(), x64.abs() @ w64.abs().t()
    bound = U[dtype] * ref.abs() + k / 16 * 2.0 ** -23 * mag
    want = ref + b.double() if bias else ref
    if bias:
        bound = bound + U[dtype] * (want.abs() + U[dtype] * ref.abs())
    y = xn.Linear(w, b)(x)
    assert bool(((y.double() - want).abs() <= bound).all())
    if not bias and n % 8 == 0:  # the same weight stored [k, n]
        y = xn.matmul(x, w.t().contiguous())
        assert bool(((y.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("m,n,k", [(1, 3100, 4096), (9, 250, 272), (32, 4096, 4112), (64, 520, 8192), (96, 4096, 2064), (128, 640, 4096),
                                   (40, 22528, 256)])
def test_e4m3_rows(xn, cuda, variant, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device=cuda).bfloat16()
    wq, ws = xn.quantize_weights_fp8(torch.randn(n, k, generator=g, device=cuda) * 0.02)
    hi, lo, xs = xn.split_rows_e4m3(x)
    f = lambda t: t.view(torch.float8_e4m3fn).double()
    a = (f(hi) + (f(lo) if variant == 0 else 0.0)) * xs.double()[:, None]
    w = f(wq) * ws.double()[:, None]
    ref, mag = a @ w.t(), (a.abs() + (f(lo).abs() * xs.double()[:, None] if variant == 0 else 0.0)) @ w.abs().t()
    y = xn.linear_fp8(x, wq, ws, variant)
    bound = 2.0 ** -8 * ref.abs() + k / 32 * 2.0 ** -22 * mag
    assert bool(((y.double() - ref).abs() <= bound).all())
