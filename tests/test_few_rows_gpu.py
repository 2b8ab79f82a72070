"""matmul of up to 16 rows with one right-hand side per batch entry or a row-major right-hand side, lhs rows at any pitch,
and the row softmax between the two products of decode attention -- at the edges of their tiles.

Bounds: an output is one rounding of an f32 sum of exact products, so |y - ref| <= u |ref| + k 2^-24 sum|a||b| with
u = 2^-8 (bf16), 2^-11 (f16), half an ulp doubled; the reference is f64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -23}


def _check(y, a, b, rhs_t):
    a64, b64 = a.double(), b.double()
    if rhs_t:
        b64 = b64.transpose(-1, -2)
    ref = a64 @ b64
    mag = a64.abs() @ b64.abs()
    err = (y.double() - ref).abs()
    assert not torch.isnan(y).any()
    assert bool((err <= U[y.dtype] * ref.abs() + a.shape[-1] * 2.0 ** -24 * mag).all()), float((err / (mag + 1e-30)).max())


def _rand(g, *shape, dtype):
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,m,n,k", [(3, 1, 17, 8), (5, 16, 130, 40), (2, 9, 64, 1032), (40, 3, 1501, 128), (300, 2, 33, 64),
                                         (2, 8, 16, 2048)])
def test_batched_rows_against_their_own_weights(xn, cuda, dtype, batch, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(batch + n)
    x = _rand(g, m, batch, k, dtype=dtype).transpose(0, 1)  # slices of a wider row
    w = _rand(g, batch, n, k, dtype=dtype)
    _check(xn.matmul_t(x, w), x, w, True)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,m,n,k", [(1, 1, 8, 16), (3, 16, 72, 33), (2, 9, 136, 1501), (1, 5, 200, 8192), (8, 1, 128, 3000),
                                         (1, 16, 64, 11264), (7, 3, 5, 16)])
def test_few_rows_against_a_row_major_right_hand_side(xn, cuda, dtype, batch, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(m + k)
    x = _rand(g, batch, m, k, dtype=dtype)
    w = _rand(g, batch, k, (n + 7) // 8 * 8, dtype=dtype)[..., :n]
    _check(xn.matmul(x, w), x, w, False)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,m,n,k", [(2, 17, 128, 1501), (3, 200, 64, 35), (1, 65, 256, 1003)])
def test_lhs_rows_off_16_byte_boundaries(xn, cuda, dtype, batch, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(m + k)
    x, w = _rand(g, batch, m, k, dtype=dtype), _rand(g, batch, k, n, dtype=dtype)
    _check(xn.matmul(x, w), x, w, False)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(3, 1), (5, 7), (4, 255), (3, 1501), (2, 4096), (3, 8191), (2, 9001)])
def test_softmax_rows_of_any_length(xn, cuda, dtype, rows, cols):
    """x - max is rounded to T, so is the exponential (relative 2u together with the argument's |x - max| u <= 12 u), and
    the quotient once more: 16 u of the value."""
    g = torch.Generator(device=cuda).manual_seed(cols)
    x = _rand(g, rows, cols, dtype=dtype)
    y = xn.ops.softmax(x)
    ref = torch.softmax(x.double(), -1)
    u = U[dtype] if dtype != torch.float32 else cols * 2.0 ** -24
    assert bool(((y.double() - ref).abs() <= 16 * u * ref + 1e-7).all())


@pytest.mark.parametrize("how", ["add", "rms_norm", "split"])
def test_a_weight_written_by_the_call_before(xn, cuda, how):
    """A Linear may fetch its weight before its dependency wait: not while the row kernel that writes it still runs.
    Inputs are small integers and the expected product is formed after a synchronisation, so both sides are equal."""
    g = torch.Generator(device=cuda).manual_seed(5)
    n, k = 22528, 4096
    a = torch.randint(-4, 5, (n, k), generator=g, device=cuda).to(torch.bfloat16)
    x = torch.randint(-4, 5, (1, k), generator=g, device=cuda).to(torch.bfloat16)
    alpha = torch.ones(k, device=cuda, dtype=torch.bfloat16)
    for _ in range(8):
        if how == "split":
            q, _, s = xn.split_rows_e4m3(a, False)
            y = xn.linear_fp8(x, q, s)
            torch.cuda.synchronize()
            ref = xn.linear_fp8(x, q, s)
        else:
            w = xn.ops.add(a, a) if how == "add" else xn.ops.rms_norm(a, alpha, 1e-5)
            y = xn.Linear(w)(x)
            torch.cuda.synchronize()
            ref = xn.Linear(w)(x)
        torch.cuda.synchronize()
        assert torch.equal(y, ref)
        a = a.roll(1, 0)
        if how == "split":
            q.zero_()
        else:
            w.zero_()
        torch.cuda.synchronize()
        del y, ref
