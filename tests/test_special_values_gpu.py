"""Rows with infinities, NaN, sums of squares that overflow and zeros without an epsilon: the vector kernels give what the scalar
ones give (which run when a pointer is off the 16-byte boundaries), element by element.

On these rows the f32 sum of squares is 0, inf or NaN in any order of addition, so both kernels have the same denominator and the
results are equal, not merely close."""
import pytest
import torch

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")


def _rows(dtype, cols, device):
    g = torch.Generator(device=device).manual_seed(cols)
    x = torch.randn(6, cols, generator=g, device=device).to(dtype)
    x[0, cols // 3] = INF
    x[1, 1] = -INF
    x[1, 5] = INF
    x[2, cols - 1] = NAN
    x[3] = 0.0
    if dtype == torch.bfloat16:  # finite, but the squares overflow
        x[4, 0] = 1e20
        x[5] = 3e38
    else:
        x[4:] = 0.0
    return x


def _off(t):
    """A copy that starts one element behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [8, 384, 4096, 8192])
def test_rms_norm(xn, cuda, dtype, cols):
    x, alpha = _rows(dtype, cols, cuda), torch.rand(cols, device=cuda).to(dtype)
    y, want = xn.ops.rms_norm(x, alpha, 0.0), xn.ops.rms_norm(_off(x), alpha, 0.0)
    torch.testing.assert_close(y, want, rtol=0, atol=0, equal_nan=True)
    assert (y[0].float().isnan().sum() == 1) and (dtype != torch.bfloat16 or (y[4:] == 0).all())


@pytest.mark.parametrize("cols", [384, 4096])
def test_pieces_of_a_normalised_sum(xn, cuda, cols):
    dtype, rows = torch.bfloat16, 6
    x, alpha = _rows(dtype, cols, cuda), torch.rand(cols, device=cuda).to(dtype)
    zero = torch.zeros_like(x)

    def run(a):
        hi, lo = (torch.empty(rows, cols, dtype=torch.uint8, device=cuda) for _ in range(2))
        xs, total = torch.empty(rows, device=cuda), torch.empty_like(x)
        xn._lib.check(xn.lib().xn_mm_add_rms_norm_split_e4m3(
            hi.data_ptr(), lo.data_ptr(), xs.data_ptr(), total.data_ptr(), a.data_ptr(), zero.data_ptr(), alpha.data_ptr(), xn.BF16, rows,
            cols, 0.0, torch.cuda.current_stream().cuda_stream))
        return hi.view(torch.float8_e4m3fn).float(), lo.view(torch.float8_e4m3fn).float(), xs, total

    for got, want in zip(run(x), run(_off(x))):
        torch.testing.assert_close(got, want, rtol=0, atol=0, equal_nan=True)
