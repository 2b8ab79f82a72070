"""What the operators refuse before anything is allocated or launched.  The checks need no device, so they run on CPU tensors."""
import pytest
import torch


@pytest.mark.parametrize("shape", [(4, 512), (4, 128), (1, 512), (2, 2, 512), (2, 3, 128), (4, 257), (512,), (128,), (4, 0), ()])
def test_int4_layer_refuses_rows_of_another_width(xn, shape):
    """Rows of 2 k elements would be twice as many rows as the output has, rows of k / 2 half as many."""
    layer = xn.LinearQ4(torch.zeros(16 * 256, dtype=torch.uint8), 16, 256)
    with pytest.raises(xn.XnError, match="rows of 256 elements"):
        layer(torch.zeros(shape))


@pytest.mark.parametrize("shape", [(4, 512), (4, 128), (2, 2, 272), (128,), ()])
def test_fp8_layer_refuses_rows_of_another_width(xn, shape):
    """Longer rows would read past the weight's end."""
    layer = xn.LinearFp8(torch.zeros(16, 256, dtype=torch.uint8), torch.ones(16))
    with pytest.raises(xn.XnError, match="rows of 256 elements"):
        layer(torch.zeros(shape, dtype=torch.bfloat16))


def test_fp8_linear_takes_a_matrix(xn):
    with pytest.raises(xn.XnError, match="a matrix"):
        xn.linear_fp8(torch.zeros(2, 3, 256, dtype=torch.bfloat16), torch.zeros(16, 256, dtype=torch.uint8), torch.ones(16))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 256), (256,), (2, 3, 256), (0, 256)])
def test_fp8_layer_takes_any_leading_dimensions(xn, cuda, shape):
    g = torch.Generator(device=cuda).manual_seed(1)
    layer = xn.LinearFp8.from_weight(torch.randn(48, 256, generator=g, device=cuda))
    x = torch.randn(*shape, generator=g, device=cuda).bfloat16()
    y = layer(x)
    assert y.shape == (*shape[:-1], 48)
    assert torch.equal(y.reshape(-1, 48), xn.linear_fp8(x.reshape(-1, 256), layer.wq, layer.ws))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 256), (256,), (2, 3, 256), (0, 256), (2, 0, 256), (0, 7)])
def test_int4_layer_takes_any_leading_dimensions(xn, cuda, shape):
    g = torch.Generator(device=cuda).manual_seed(1)
    layer = xn.LinearQ4.from_weight(torch.randn(48, 256, generator=g, device=cuda))
    x = torch.randn(*shape, generator=g, device=cuda)
    y = layer(x)
    assert y.shape == (*shape[:-1], 48)
    if x.numel():
        xq, xs = xn.quantize_rows_i8(x.reshape(-1, 256))
        assert torch.equal(y.reshape(-1, 48), xn.linear_q4(xq, xs, layer.wq, 48))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float64, torch.int64, torch.int32, torch.int8, torch.uint8])
def test_refused_types_are_named_as_torch_names_them(xn, cuda, dtype):
    a = torch.zeros(4, 4, dtype=dtype, device=cuda)
    with pytest.raises(xn.XnError, match=f"not supported for dtype {dtype}"):
        xn.matmul_t(a, a)


@pytest.mark.gpu
def test_add_of_transposed_views(xn, cuda):
    a, b = torch.randn(37, 50, device=cuda), torch.randn(37, 50, device=cuda)
    for x, y in ((a.t(), b.t()), (a.t(), b.t().contiguous()), (a.t().contiguous(), b.t())):
        assert torch.equal(xn.ops.add(x, y), x + y)
    with pytest.raises(xn.XnError):
        xn.ops.add(a, b[:5])
