"""Softmax of rows that share a CTA, a warp each: row counts around a CTA's and lengths around a warp's share of vectors, rows that start
anywhere.

Bound: x - max is rounded to T, so is the exponential (relative 2u together with the argument's |x - max| u <= 12 u), and the
quotient once more: 16 u of the value; f32 sums of at most 520 terms, 520 2^-24."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,u", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11), (torch.float32, 520 * 2.0 ** -24)])
@pytest.mark.parametrize("rows", [1, 2, 3, 9, 1183, 1184, 1193, 9475])
@pytest.mark.parametrize("cols", [1, 8, 15, 33, 127, 128, 255, 256, 263, 264, 511, 512, 519, 520])
def test_against_f64(xn, cuda, dtype, u, rows, cols):
    g = torch.Generator(device=cuda).manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=g, device=cuda).to(dtype)
    y, ref = xn.ops.softmax(x), torch.softmax(x.double(), -1)
    assert bool(((y.double() - ref).abs() <= 16 * u * ref + 1e-7).all())


def test_rows_without_a_finite_maximum(xn, cuda):
    """As torch has it: a row of -inf, or with +inf or NaN in it, is NaN where the exponentials are; its neighbours are not touched."""
    x = torch.zeros(5, 40, device=cuda)
    x[1] = -float("inf")
    x[3, 7] = float("nan")
    y = xn.ops.softmax(x)
    for r in (0, 2, 4):
        assert torch.equal(y[r], torch.full((40,), 1 / 40, device=cuda))
    assert y[1].isnan().all() and y[3].isnan().all()
