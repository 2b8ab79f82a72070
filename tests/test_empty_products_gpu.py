"""A product over no elements is zeros (plus a bias), on every route: few rows, many rows, batches, both right-hand side layouts,
slices of live tensors, and the C entry point itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("lead", [(1,), (7,), (16,), (40,), (100,), (300,), (3, 1), (3, 16), (2, 3, 5), (2, 40)])
def test_slices_without_elements(xn, cuda, dtype, lead):
    x, w = torch.ones(*lead, 64, dtype=dtype, device=cuda), torch.ones(*lead[:-1], 512, 64, dtype=dtype, device=cuda)
    for off in (0, 16):
        xe, we = x[..., off:off], w[..., off:off]
        for rhs, t in ((we, True), (we.transpose(-1, -2), False), (w.transpose(-1, -2)[..., off:off, :], False),
                       (torch.ones(*lead[:-1], 64, 512, dtype=dtype, device=cuda)[..., off:off, :], False)):
            y = torch.full((*lead, 512), float("nan"), dtype=dtype, device=cuda)
            xn.matmul_(y, xe, rhs, t)
            assert (y == 0).all()


@pytest.mark.parametrize("dtype,code", [(torch.bfloat16, 2), (torch.float16, 1), (torch.float32, 0)])
@pytest.mark.parametrize("batch,m,n", [(1, 1, 64), (1, 16, 4096), (1, 64, 300), (1, 300, 300), (4, 3, 130), (4, 70, 96)])
@pytest.mark.parametrize("rhs_rows", [True, False])
def test_c_entry(xn, cuda, dtype, code, batch, m, n, rhs_rows):
    a = torch.ones(4096, dtype=dtype, device=cuda)
    y = torch.full((batch, m, n), float("nan"), dtype=dtype, device=cuda)
    rhs_cs, rhs_rs = (8, 1) if rhs_rows else (1, (n + 7) // 8 * 8)
    xn._lib.check(xn.lib().xn_mm_gemm(code, y.data_ptr(), a.data_ptr(), 0, a.data_ptr(), 0, m, n, 0, batch, 8, 8, 1, n, 1, 8, rhs_cs,
                                      rhs_rs, torch.cuda.current_stream().cuda_stream))
    assert (y == 0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [1, 40])
def test_layer_without_inputs_is_its_bias(xn, cuda, dtype, rows):
    w, b = torch.ones(128, 64, dtype=dtype, device=cuda), torch.randn(128, device=cuda).to(dtype)
    y = xn.Linear(w[:, :0], b)(torch.ones(rows, 64, dtype=dtype, device=cuda)[:, :0])
    assert torch.equal(y, b.expand(rows, 128))
