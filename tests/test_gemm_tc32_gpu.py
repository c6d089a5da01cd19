"""fp32 MatMul on the tensor cores and in 32 x 32 CUDA-core tiles (rg_b200_mat_mul with force_kernel = 5 and 6 and the automatic
route) against fp64.

Every element within the bound of a sum of k fp32 products in any order, (k + 16) 2^-24 of the sum of their magnitudes,
and the 2-norm of the error within that of the CUDA-core kernel on the same data (or 1.2e-7 = one rounding of the result, where
k is so small that the kernel's error is below it)."""
import pytest
import torch

from refactorgraph_b200 import capi

import _ops as ops

pytestmark = pytest.mark.gpu


def _err(y, want):
    return float((y.double() - want).norm() / want.norm())


@pytest.mark.parametrize("force", [5, 6])
@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("batch,m,n,k", [(1, 1, 1, 1), (1, 7, 130, 100), (1, 32, 4096, 1024), (1, 33, 1000, 2752), (1, 64, 36, 64), (1, 65, 300, 509),
                                         (1, 128, 128, 64), (1, 129, 127, 65), (1, 509, 1024, 1024), (3, 100, 509, 64), (5, 77, 64, 509), (4, 32, 32, 64),
                                         (1, 300, 5000, 2752), (2, 513, 261, 130), (1, 700, 300, 11008)])
def test_against_fp64_and_the_cuda_core_kernel(force, trans_b, batch, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m * 3 + n + k)
    a = torch.randn(batch, m, k, device="cuda", generator=g)
    b = torch.randn(batch, *((n, k) if trans_b else (k, n)), device="cuda", generator=g)
    c = torch.randn(n, device="cuda", generator=g)
    if batch == 1:
        a, b = a[0], b[0]
    bt = b.double().transpose(-1, -2) if trans_b else b.double()
    prod = a.double() @ bt
    y = ops.mat_mul(a, b, trans_b=trans_b, force=force)
    assert capi.load().rg_b200_error_state() == 0
    bound = (k + 16) * 2.0 ** -24 * (a.double().abs() @ bt.abs())
    assert bool(((y.double() - prod).abs() <= bound).all())
    simt = ops.mat_mul(a, b, trans_b=trans_b, force=1)
    assert _err(y, prod) <= max(1.02 * _err(simt, prod), 1.2e-7)
    assert torch.equal(y, ops.mat_mul(a, b, trans_b=trans_b, force=force))  # fixed order of summation
    y2 = ops.mat_mul(a, b, c, trans_b=trans_b, alpha=0.5, beta=2.0, force=force)
    want = 0.5 * prod + 2.0 * c.double()
    assert bool(((y2.double() - want).abs() <= 0.5 * bound + 2.0 ** -23 * (want.abs() + 2.0 * c.double().abs())).all())


@pytest.mark.parametrize("force", [5, 6])
def test_shared_operand_of_a_batch_and_unaligned_operands(force):
    g = torch.Generator(device="cuda").manual_seed(5)
    a, b = torch.randn(4, 70, 96, device="cuda", generator=g), torch.randn(96, 200, device="cuda", generator=g)
    torch.testing.assert_close(ops.mat_mul(a, b, force=force).double(), a.double() @ b.double(), atol=3e-5, rtol=1e-5)
    a, b = b.T.contiguous(), torch.randn(3, 96, 40, device="cuda", generator=g)
    torch.testing.assert_close(ops.mat_mul(a, b, force=force).double(), a.double() @ b.double(), atol=3e-5, rtol=1e-5)
    for m in (40, 100):
        a, b = torch.randn(m * 96 + 1, device="cuda", generator=g)[1:].view(m, 96), torch.randn(96 * 200 + 3, device="cuda", generator=g)[3:].view(96, 200)
        torch.testing.assert_close(ops.mat_mul(a, b, force=force).double(), a.double() @ b.double(), atol=3e-5, rtol=1e-5)


@pytest.mark.parametrize("force", [0, 5, 6])
@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("k", [1, 2, 3, 5, 8, 16, 24, 64, 100])
def test_short_sums_are_as_close_as_fused_multiply_adds(force, trans_b, k):
    """With few terms a product's own rounding is nearly all the error there is.  What the tensor-core form leaves out is at most 2^-24 of a
    product and may show beside the one rounding of a sum of one (which the automatic route leaves to the CUDA cores); 2 % are for
    the luck of the data."""
    for m in (20, 64, 300):
        g = torch.Generator(device="cuda").manual_seed(k + m)
        a = torch.randn(m, k, device="cuda", generator=g)
        b = torch.randn(*((1000, k) if trans_b else (k, 1000)), device="cuda", generator=g)
        want = a.double() @ (b.double().T if trans_b else b.double())
        simt, y = ops.mat_mul(a, b, trans_b=trans_b, force=1), ops.mat_mul(a, b, trans_b=trans_b, force=force)
        assert _err(y, want) <= (1.06 if k == 1 and force == 5 else 1.02) * _err(simt, want)
        if k == 1:
            assert bool(((y.double() - want).abs() <= 2.0 ** -23 * want.abs()).all())


@pytest.mark.parametrize("force", [5, 6])
@pytest.mark.parametrize("m", [20, 60, 200])
@pytest.mark.parametrize("k", [8, 300])
@pytest.mark.parametrize("exponent", [-100, -110, -116, -120, -126, -133, -140, 120])
def test_small_and_large_operands(force, m, k, exponent):
    """One operand around 2^exponent (subnormal numbers from -126 down), the other the size that makes the result ordinary."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    for swap in (False, True):
        scale = (2.0 ** (-exponent // 2), 2.0 ** exponent) if swap else (2.0 ** exponent, 2.0 ** (-exponent // 2))
        a = (torch.rand(m, k, device="cuda", generator=g, dtype=torch.float64) * scale[0]).float()
        b = (torch.rand(k, 132, device="cuda", generator=g, dtype=torch.float64) * scale[1]).float()
        want = a.double() @ b.double()
        simt, y = ops.mat_mul(a, b, force=1), ops.mat_mul(a, b, force=force)
        assert _err(y, want) <= 1.02 * _err(simt, want)
        assert bool(((y.double() - want).abs() <= (k + 16) * 2.0 ** -24 * want).all())


@pytest.mark.parametrize("force", [5, 6])
@pytest.mark.parametrize("m", [20, 60, 200])
def test_results_that_are_subnormal(force, m):
    """Products of 2^-140: no further off than a quantum (2^-149) a rounding, as a chain of fp32 multiply-adds."""
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = (2.0 ** -70 * torch.randn(*s, device="cuda", generator=g) for s in ((m, 200), (200, 132)))
    want = a.double() @ b.double()
    simt, y = ops.mat_mul(a, b, force=1), ops.mat_mul(a, b, force=force)
    assert _err(y, want) <= 1.02 * _err(simt, want)


@pytest.mark.parametrize("force", [5, 6])
@pytest.mark.parametrize("m", [20, 60, 200])
def test_infinity_times_the_smallest_numbers(force, m):
    """inf x 2^-149 is inf, inf x 0 is NaN, and sums that stay below the largest number stay finite."""
    a, b = torch.ones(m, 72, device="cuda"), torch.ones(72, 140, device="cuda")
    a[3, 70], a[m - 1, 5] = float("inf"), float("-inf")
    b[70, 4], b[70, 5], b[5, 139] = 2.0 ** -149, 0.0, 2.0 ** -140
    y, want = ops.mat_mul(a, b, force=force), ops.mat_mul(a, b, force=1)
    assert want[3, 4] == float("inf") and want[3, 5].isnan() and want[m - 1, 139] == float("-inf")
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y[~y.isnan()], want[~want.isnan()])
    a, b = torch.full((m, 2), 2.0 ** 63, device="cuda"), torch.full((2, 140), 2.0 ** 63 * (2 - 2.0 ** -10), device="cuda")
    assert torch.equal(ops.mat_mul(a, b, force=force).double(), a.double() @ b.double())
    a, b = torch.full((m, 1), 2.0 ** 64 * (1 - 2.0 ** -24), device="cuda"), torch.full((1, 140), 2.0 ** 64 * (1 - 2.0 ** -24), device="cuda")
    assert torch.equal(ops.mat_mul(a, b, force=force).double(), torch.full((m, 140), 2.0 ** 128 * (1 - 2.0 ** -23), device="cuda", dtype=torch.float64))
    c = torch.randn(m, 140, device="cuda")
    assert torch.equal(ops.mat_mul(a, b, c, alpha=0.5, beta=2.0, force=force), ops.mat_mul(a, b, c, alpha=0.5, beta=2.0, force=1))


@pytest.mark.parametrize("force", [5, 6])
@pytest.mark.parametrize("m", [60, 200])
def test_values_at_the_ends_of_the_range(force, m):
    """Infinities, NaNs, the largest finite values, zeros and exact small integers give what the CUDA-core kernel gives."""
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = torch.randint(-3, 4, (m, 160), device="cuda", generator=g).float(), torch.randint(-3, 4, (160, 130), device="cuda", generator=g).float()
    assert torch.equal(ops.mat_mul(a, b, force=force).double(), a.double() @ b.double())
    top = torch.finfo(torch.float32).max
    for value in (float("inf"), float("-inf"), float("nan"), top, -top):
        x = a.clone()
        x[7, 3], x[m - 3, 159], b[3, 5] = value, value, 0.0
        y, want = ops.mat_mul(x, b, force=force), ops.mat_mul(x, b, force=1)
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
        ok = want.isfinite()
        torch.testing.assert_close(y[ok], want[ok], atol=1e-5, rtol=1e-6)
        w = b.clone()
        w[11, 64] = value
        y, want = ops.mat_mul(a, w, force=force), ops.mat_mul(a, w, force=1)
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())


@pytest.mark.parametrize("batch,m,n,k,trans_a", [(1, 64, 1024, 1024, False), (16, 64, 64, 64, False), (1, 2, 100, 100, False), (1, 64, 32000, 1024, False), (1, 509, 2752, 1024, False), (1, 128, 1024, 1024, True)])
def test_the_automatic_route_agrees(batch, m, n, k, trans_a):
    """Both sides of the dispatch line, and what the tensor-core form does not take."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(batch, *((k, m) if trans_a else (m, k)), device="cuda", generator=g)
    b = torch.randn(batch, k, n, device="cuda", generator=g)
    y = ops.mat_mul(a, b, trans_a=trans_a)
    want = (a.transpose(-1, -2) if trans_a else a).double() @ b.double()
    assert _err(y, want) <= 1e-6
