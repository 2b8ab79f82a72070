"""A Linear may fetch its weight before its dependency wait: not while the matmul of a few rows that writes the weight still runs (a
[k, n] or a batched right-hand side); the layer either follows at once or behind a kernel that announces itself early.

Inputs are small integers and the reference is formed after a synchronisation, so both sides are equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ints(g, *shape, dtype):
    return torch.randint(-2, 3, shape, generator=g, device="cuda").to(dtype)


# weight [n, k] of the layer as a product: batch, rows, columns, depth, right-hand side transposed
@pytest.mark.parametrize("dtype,batch,m,n,k,rhs_t", [
    (torch.bfloat16, 64, 16, 2048, 512, False), (torch.bfloat16, 300, 5, 1024, 256, False), (torch.float16, 1024, 2, 1032, 136, False),
    (torch.bfloat16, 64, 16, 2048, 512, True), (torch.bfloat16, 300, 5, 1024, 256, True), (torch.float16, 1024, 2, 1032, 136, True)])
@pytest.mark.parametrize("between", [False, True])
def test_a_weight_written_by_a_matmul(xn, cuda, dtype, batch, m, n, k, rhs_t, between):
    g = torch.Generator(device=cuda).manual_seed(m + n)
    a = _ints(g, batch, m, k, dtype=dtype)
    b = _ints(g, batch, *((n, k) if rhs_t else (k, n)), dtype=dtype) if batch > 1 else _ints(g, *((n, k) if rhs_t else (k, n)), dtype=dtype)
    x = _ints(g, 1, n, dtype=dtype)
    other = torch.randn(4, 256, device=cuda)
    for _ in range(8):
        w = xn.matmul_with_t(a, b, rhs_t).view(batch * m, n)
        if between:
            xn.quantize_rows_i8(other)
        y = xn.Linear(w)(x)
        torch.cuda.synchronize()
        ref = xn.Linear(w)(x)
        torch.cuda.synchronize()
        assert torch.equal(y, ref)
        w.zero_()
        a = a.roll(1, 1)
        torch.cuda.synchronize()
        del y, ref, w
