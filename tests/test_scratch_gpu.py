"""What the library keeps for itself, and what happens when there is none of it: a context that grows by one key per call, a first call
under capture, an operand too large to be copied."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_growing_context_does_not_pile_up_scratch(xn, cuda):
    """p.v over rows off 16-byte boundaries copies the rows to scratch, a little more of it for every few keys: replaced blocks are kept
    until they are released, so a block grows by half at least and the kept ones stay below twice the block in use."""
    b, m, n, lo, hi = 16, 64, 64, 2001, 2401
    p = torch.randn(b, m, 3001, device=cuda).bfloat16()
    v = torch.randn(b, hi, n, device=cuda).bfloat16()
    y = torch.empty(b, m, n, device=cuda, dtype=torch.bfloat16)
    xn.matmul_(y, p[..., :lo], v[:, :lo], False)
    torch.cuda.synchronize()
    xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
    free0 = torch.cuda.mem_get_info()[0]
    for k in range(lo, hi):
        xn.matmul_(y, p[..., :k], v[:, :k], False)
    torch.cuda.synchronize()
    used = free0 - torch.cuda.mem_get_info()[0]
    largest = 2 * b * m * ((hi + 7) // 8 * 8)
    assert used <= 4.5 * largest + (16 << 20), used  # 1.5 in use, below 3 kept, pages
    ref = p[..., :hi - 1].double() @ v[:, :hi - 1].double()
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 0.02).all())
    xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
