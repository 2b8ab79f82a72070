"""Decode steps back to back through the SAME activation buffers: the quantizer announces the linear before it has written, so the
linear's blocks start beside the previous step's and must read the new codes and scales all the same.

Block sums are integers and the f32 sums run in a fixed order: results are equal to those of steps taken one at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("m,n,k", [(1, 4096, 4096), (4, 11264, 4096), (16, 11264, 4096), (16, 4096, 11264), (9, 2064, 14336), (8, 20, 16384),
                                   (7, 40000, 256)])
def test_steps_through_one_pair_of_buffers(xn, cuda, bits, m, n, k):
    g = torch.Generator(device=cuda).manual_seed(m + n)
    w = torch.randn(n, k, generator=g, device=cuda) * 0.02
    wq = (xn.quantize_weights_q4 if bits == 4 else xn.quantize_weights_q8)(w)
    linear = xn.linear_q4 if bits == 4 else xn.linear_q8
    xs = [torch.randn(m, k, generator=g, device=cuda) * (i + 1) for i in range(6)]
    want = []
    for x in xs:
        q, s = xn.quantize_rows_i8(x)
        torch.cuda.synchronize()
        want.append(linear(q, s, wq, n))
        torch.cuda.synchronize()
    pair = (torch.empty(m, k, dtype=torch.int8, device=cuda), torch.empty(m, device=cuda))
    for _ in range(20):
        got = []
        for x in xs:
            q, s = xn.quantize_rows_i8(x, out=pair)
            got.append(linear(q, s, wq, n))
        torch.cuda.synchronize()
        for y, z in zip(got, want):
            assert torch.equal(y, z)
