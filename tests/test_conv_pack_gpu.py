"""conv1d / conv_transpose1d on the tensor-memory path at the edges of the repacking launch: channels and positions that do not
fill a block, one tap and more taps than a block's tile holds (then the taps are repacked by launches of their own), batches.

Bound: 16-bit, one rounding of an f32 sum of exact products, u |ref| + K 2^-23 sum|x||w|; f32, products to 2^-21 and sums in
f32, (2^-20 + K 2^-24) sum|x||w|; one more rounding for the bias.  The reference is f64."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

U = {torch.float32: 2.0 ** -23, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tr,batch,ci,co,length,ks,stride,pad", [
    (False, 1, 8, 5, 1, 1, 1, 0), (False, 3, 72, 33, 31, 3, 1, 1), (False, 2, 136, 130, 65, 7, 2, 0), (False, 1, 512, 512, 64, 7, 1, 3),
    (False, 1, 16, 24, 400, 201, 3, 5), (True, 1, 16, 9, 5, 4, 2, 0), (True, 2, 200, 64, 33, 10, 5, 1), (True, 1, 8, 16, 70, 180, 90, 0)])
def test_against_f64(xn, cuda, dtype, tr, batch, ci, co, length, ks, stride, pad):
    g = torch.Generator(device=cuda).manual_seed(ci + ks)
    x = torch.randn(batch, ci, length, generator=g, device=cuda).to(dtype)
    w = torch.randn(*((ci, co, ks) if tr else (co, ci, ks)), generator=g, device=cuda).to(dtype)
    b = torch.randn(co, generator=g, device=cuda).to(dtype)
    f = F.conv_transpose1d if tr else F.conv1d
    ref = f(x.double(), w.double(), b.double(), stride=stride, padding=pad)
    mag = f(x.double().abs(), w.double().abs(), b.double().abs(), stride=stride, padding=pad)
    y = (xn.ops.conv_transpose1d if tr else xn.ops.conv1d)(x, w, b, stride, pad, *((0, 1) if tr else (1, 1)))
    assert y.shape == ref.shape and not torch.isnan(y).any()
    lim = (2.0 ** -20 + ci * ks * 2.0 ** -24) * mag if dtype == torch.float32 else 2 * U[dtype] * (ref.abs() + b.double().abs()[:, None]) + ci * ks * 2.0 ** -23 * mag
    assert bool(((y.double() - ref).abs() <= lim).all())
