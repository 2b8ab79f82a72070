"""What the library keeps for itself: a context that grows by one key per call, a first call under capture, an operand too large to be
copied."""
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


def test_rows_off_16_byte_boundaries_under_capture(xn, cuda):
    """The first call of its kind may be a captured one."""
    xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
    g = torch.Generator(device=cuda).manual_seed(2)
    x = torch.randn(3, 70, 1003, generator=g, device=cuda).bfloat16()
    w = torch.randn(3, 1003, 72, generator=g, device=cuda).bfloat16()
    y = torch.zeros(3, 70, 72, device=cuda, dtype=torch.bfloat16)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        xn.matmul_(y, x, w, False)
    for _ in range(2):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        ref, mag = x.double() @ w.double(), x.double().abs() @ w.double().abs()
        assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1003 * 2.0 ** -24 * mag).all())


def test_rows_too_many_to_be_copied(xn, cuda):
    """Above half a GB of rows the any-stride kernel takes the product."""
    m, n, k = 1 << 17, 8, 2049
    x = torch.randint(-2, 3, (m, k), device=cuda, dtype=torch.int8).half()
    w = torch.randint(-2, 3, (k, n), device=cuda, dtype=torch.int8).half()
    xn._lib.check(xn.lib().xn_mm_release_scratch(None, 1))
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    y = torch.empty(m, n, device=cuda, dtype=torch.float16)
    xn.matmul_(y, x, w, False)
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < 64 << 20
    for r in (slice(0, 64), slice(m - 64, m)):  # sums of small integers: exact in f32, one rounding to f16
        assert torch.equal(y[r], (x[r].double() @ w.double()).half())
