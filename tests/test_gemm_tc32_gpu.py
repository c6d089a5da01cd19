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
