"""tcgen05/TMEM GEMM (rg_b200_mat_mul with force_kernel = 3 and the automatic route) against the oracle.
fp16/bf16 operands, fp32 accumulation: max-abs 2e-2 / relative 1e-2 against fp64 on the rounded inputs; exact on
small-integer data.  Large cases use a torch fp32 matmul of the same rounded inputs as the reference."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as onp
from refactorgraph_b200 import capi

import _ops as ops

pytestmark = pytest.mark.gpu
HALF = [torch.float16, torch.bfloat16]


def _ok():
    return capi.load().rg_b200_error_state() == 0


def test_smallest_tile_exact():
    # one 128x128 tile, one k-block, integer data: exact in fp32 accumulation
    rng = np.random.default_rng(0)
    a = rng.integers(-3, 4, (128, 64)).astype(np.float32)
    b = rng.integers(-3, 4, (128, 64)).astype(np.float32)
    y = ops.mat_mul(ops.dev(a).half(), ops.dev(b).half(), trans_b=True, force=3)
    assert _ok(), "a bounded wait expired inside the tensor-core kernel"
    np.testing.assert_array_equal(y.float().cpu().numpy(), a @ b.T)


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (256, 512, 1024), (100, 300, 72), (129, 257, 4096), (512, 128, 256), (64, 64, 64)])
def test_against_numpy_oracle(dtype, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(dtype)
    b = torch.from_numpy((0.05 * rng.standard_normal((n, k))).astype(np.float32)).to(dtype)
    y = ops.mat_mul(a.cuda(), b.cuda(), trans_b=True, force=3)
    assert _ok()
    want = onp.mat_mul(a.float().numpy(), b.float().numpy(), trans_b=True)
    np.testing.assert_allclose(y.float().cpu().numpy(), want, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("trans_b", [True, False])
@pytest.mark.parametrize("m,n,k", [(512, 256, 64), (1024, 768, 512), (600, 300, 200), (513, 1000, 4096), (2050, 256, 1032), (1100, 4104, 1032)])
def test_pairs_of_ctas(dtype, trans_b, m, n, k):
    """Two CTAs share a 256 x 256 tile (tcgen05 ... cta_group::2; force_kernel = 7), ragged edges included, weights in either order;
    with a residual, alpha and beta; the second call must give the same bits."""
    n = n if trans_b else (n + 7) // 8 * 8
    rng = np.random.default_rng(m * 7 + n + k)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(dtype)
    b = torch.from_numpy((0.05 * rng.standard_normal((n, k) if trans_b else (k, n))).astype(np.float32)).to(dtype)
    c = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32)).to(dtype)
    y = ops.mat_mul(a.cuda(), b.cuda(), trans_b=trans_b, force=7)
    assert _ok()
    want = onp.mat_mul(a.float().numpy(), b.float().numpy(), trans_b=trans_b)
    np.testing.assert_allclose(y.float().cpu().numpy(), want, atol=2e-2, rtol=1e-2)
    y2 = ops.mat_mul(a.cuda(), b.cuda(), c.cuda(), trans_b=trans_b, alpha=0.5, beta=2.0, force=7)
    assert _ok()
    want2 = onp.mat_mul(a.float().numpy(), b.float().numpy(), c.float().numpy(), trans_b=trans_b, alpha=0.5, beta=2.0)
    np.testing.assert_allclose(y2.float().cpu().numpy(), want2, atol=4e-2, rtol=1e-2)
    assert torch.equal(y, ops.mat_mul(a.cuda(), b.cuda(), trans_b=trans_b, force=7))


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("m,n,k", [(1, 4096, 512), (4, 1032, 64), (7, 1000, 1032), (33, 22016, 512), (64, 128, 72), (65, 64, 64), (100, 304, 72),
                                   (129, 136, 4096), (300, 4096, 1024), (511, 256, 200), (512, 264, 64), (700, 1000, 4096)])
def test_weights_stored_k_by_n(dtype, m, n, k):
    """trans_b = 0: the weights enter as an MN-major operand (on either side of the instruction).  Integer
    data is exact in fp32 accumulation; the tolerance of the random data is the one of the K-major products."""
    rng = np.random.default_rng(m + 3 * n + k)
    a = rng.integers(-3, 4, (m, k)).astype(np.float32)
    b = rng.integers(-1, 2, (k, n)).astype(np.float32)
    yt = ops.mat_mul(ops.dev(a).to(dtype), ops.dev(b).to(dtype), force=3)
    assert _ok()
    assert torch.equal(yt.cpu(), torch.from_numpy(a @ b).to(dtype))
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(dtype)
    b = torch.from_numpy((0.05 * rng.standard_normal((k, n))).astype(np.float32)).to(dtype)
    c = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32)).to(dtype)
    y2 = ops.mat_mul(a.cuda(), b.cuda(), c.cuda(), alpha=0.5, beta=2.0, force=3)
    assert _ok()
    want = onp.mat_mul(a.float().numpy(), b.float().numpy(), c.float().numpy(), alpha=0.5, beta=2.0)
    np.testing.assert_allclose(y2.float().cpu().numpy(), want, atol=4e-2, rtol=1e-2)


@pytest.mark.parametrize("dtype", HALF)
def test_pairs_of_ctas_bias_vector_and_batch(dtype):
    """The pair kernel behind the batched call with a broadcast bias row."""
    rng = np.random.default_rng(11)
    a = torch.from_numpy(rng.standard_normal((2, 520, 128)).astype(np.float32)).to(dtype)
    b = torch.from_numpy((0.1 * rng.standard_normal((2, 264, 128))).astype(np.float32)).to(dtype)
    c = torch.from_numpy(rng.standard_normal((264,)).astype(np.float32)).to(dtype)
    y = ops.mat_mul(a.cuda(), b.cuda(), c.cuda(), trans_b=True, alpha=0.5, beta=2.0, force=7)
    assert _ok()
    want = onp.mat_mul(a.float().numpy(), b.float().numpy(), c.float().numpy(), trans_b=True, alpha=0.5, beta=2.0)
    np.testing.assert_allclose(y.float().cpu().numpy(), want, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("dtype", HALF)
def test_alpha_beta_bias_and_batch(dtype):
    rng = np.random.default_rng(7)
    a = torch.from_numpy(rng.standard_normal((3, 130, 128)).astype(np.float32)).to(dtype)
    b = torch.from_numpy((0.1 * rng.standard_normal((3, 200, 128))).astype(np.float32)).to(dtype)
    c = torch.from_numpy(rng.standard_normal((200,)).astype(np.float32)).to(dtype)
    y = ops.mat_mul(a.cuda(), b.cuda(), c.cuda(), trans_b=True, alpha=0.5, beta=2.0, force=3)
    assert _ok()
    want = onp.mat_mul(a.float().numpy(), b.float().numpy(), c.float().numpy(), trans_b=True, alpha=0.5, beta=2.0)
    np.testing.assert_allclose(y.float().cpu().numpy(), want, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("m,n,k", [(16, 4096, 4096), (32, 11008, 4096), (64, 4096, 11008), (5, 1000, 512)])
def test_skinny_swapped_operands(dtype, m, n, k):
    rng = np.random.default_rng(m * n)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(dtype).cuda()
    b = torch.from_numpy((0.02 * rng.standard_normal((n, k))).astype(np.float32)).to(dtype).cuda()
    y = ops.mat_mul(a, b, trans_b=True, force=3)
    assert _ok()
    want = a.float() @ b.float().T
    torch.testing.assert_close(y.float(), want, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("trans_b", [True, False])
@pytest.mark.parametrize("m,n,k", [(1, 4096, 64), (8, 520, 128), (9, 520, 200), (32, 256, 512), (33, 1024, 1024), (64, 1280, 8192), (48, 12288, 4096), (3, 5000, 4096)])
def test_skinny_clusters_share_a_tile(dtype, trans_b, m, n, k):
    """k divided over clusters of 1, 2, 4 and 8 CTAs, several tiles per cluster, ragged tiles and tokens; integer data is exact in
    fp32 accumulation whatever the order of the sums."""
    rng = np.random.default_rng(m + n + k)
    a, b, c = (rng.integers(-2, 3, s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    bd = ops.dev(b.T.copy() if trans_b else b).to(dtype)
    want = torch.from_numpy(a @ b + 2 * c).to(dtype)
    for _ in range(2):
        y = ops.mat_mul(ops.dev(a).to(dtype), bd, ops.dev(c).to(dtype), trans_b=trans_b, beta=2.0, force=3)
        assert _ok()
        assert torch.equal(y.cpu(), want)


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("trans_b", [True, False])
@pytest.mark.parametrize("m,n,k", [(65, 136, 2048), (100, 1024, 1024), (128, 256, 8192), (300, 2752, 1024), (333, 4096, 1024), (511, 1000, 520), (600, 520, 512)])
def test_wide_clusters_share_a_tile(dtype, trans_b, m, n, k):
    """More than 64 tokens and fewer tiles than SMs: k divided over clusters, the sums exchanged through the ring; exact integer data,
    ragged edges, residual and bias row."""
    rng = np.random.default_rng(m + n + k)
    a, b, c, r = (rng.integers(-2, 3, s).astype(np.float32) for s in ((m, k), (k, n), (m, n), (n,)))
    bd = ops.dev(b.T.copy() if trans_b else b).to(dtype)
    for add in (c, r, c):
        y = ops.mat_mul(ops.dev(a).to(dtype), bd, ops.dev(add).to(dtype), trans_b=trans_b, beta=2.0, force=3)
        assert _ok()
        assert torch.equal(y.cpu(), torch.from_numpy(a @ b + 2 * add).to(dtype))


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("m,n,k,residual", [(16, 22016, 4096, False), (32, 32000, 4096, True), (8, 20000, 4104, False)])
def test_skinny_products_of_several_tiles_a_cluster(dtype, m, n, k, residual):
    """Skinny products with more tiles than clusters: the exchange of a tile's sums overlaps the stream of the next, the receive
    buffers are used again.  The last case has a ragged last row tile and a partial last k-block."""
    rng = np.random.default_rng(m + n + k)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(dtype).cuda()
    b = torch.from_numpy((0.02 * rng.standard_normal((n, k))).astype(np.float32)).to(dtype).cuda()
    want = a.float() @ b.float().T
    if residual:
        c = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32)).to(dtype).cuda()
        y = ops.mat_mul(a, b, c=c, trans_b=True, force=3)
        want = want + c.float()
    else:
        y = ops.mat_mul(a, b, trans_b=True, force=3)
    assert _ok()
    torch.testing.assert_close(y.float(), want, atol=2e-2, rtol=1e-2)
    y2 = ops.mat_mul(a, b, c=c, trans_b=True, force=3) if residual else ops.mat_mul(a, b, trans_b=True, force=3)
    assert torch.equal(y, y2)          # fixed summation order: a second call gives the same bits


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("trans_b", [True, False])
@pytest.mark.parametrize("m,n,k", [(70, 256, 64), (333, 4096, 1024), (1100, 4104, 1032), (40, 1024, 512)])
def test_addend_that_starts_off_a_16_byte_boundary(dtype, trans_b, m, n, k):
    """C may start at any element (a bias row, a residual, the matrices of a batch at any distance): it is then read element by
    element, in the plain epilogue, behind clusters and on CTA pairs.  Integer data, exact."""
    rng = np.random.default_rng(m + n + k)
    a, b = rng.integers(-2, 3, (m, k)).astype(np.float32), rng.integers(-2, 3, (k, n)).astype(np.float32)
    ad, bd = ops.dev(a).to(dtype), ops.dev(b.T.copy() if trans_b else b).to(dtype)
    prod = ad.float() @ (bd.float().T if trans_b else bd.float())
    assert torch.equal(prod.cpu(), torch.from_numpy(a @ b))
    for shape in ((n,), (m, n)):
        for off in (1, 4, 8):
            c = torch.randint(-2, 3, (int(np.prod(shape)) + off,), device="cuda").to(dtype)[off:].view(shape)
            y = ops.mat_mul(ad, bd, c, trans_b=trans_b, beta=2.0, force=3)
            assert _ok()
            assert torch.equal(y, (prod + 2 * c.float()).to(dtype))
    if not trans_b and m * n * k < 2 ** 26:
        return  # a batch of small products with weights [k, n] is not tcgen05's
    p = capi.MatMulParams()
    p.dtype, p.m, p.n, p.k, p.trans_b, p.alpha, p.beta, p.batch = ops.DT[dtype], m, n, k, int(trans_b), 1.0, 1.0, 2
    p.stride_y, p.has_bias, p.bias_row_stride, p.bias_col_stride, p.stride_c, p.force_kernel = m * n, 1, n, 1, m * n + 3, 3
    c, y = torch.randint(-2, 3, (2 * (m * n + 3),), device="cuda").to(dtype), torch.empty(2, m, n, dtype=dtype, device="cuda")
    capi.call("mat_mul", p, [ad.data_ptr(), bd.data_ptr(), c.data_ptr()], [y.data_ptr()], stream=torch.cuda.current_stream().cuda_stream)
    assert torch.equal(y, (prod + c.view(2, -1)[:, :m * n].view(2, m, n).float()).to(dtype))


@pytest.mark.parametrize("dtype", HALF)
@pytest.mark.parametrize("m,n,k,force", [(4, 12288, 4096, 2), (9, 256, 8192, 4), (16, 128, 4096, 4), (8, 256, 8192, 4)])
def test_the_automatic_route_of_products_too_small_for_tcgen05(dtype, m, n, k, force):
    """Few rows against few weight rows (less than 64 x 64 results), or a result off a 16-byte boundary, are not left to the CUDA cores
    where a streaming kernel takes them: the automatic route gives that kernel's bits."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, b = torch.randn(m, k, device="cuda", generator=g).to(dtype), torch.randn(n, k, device="cuda", generator=g).to(dtype)
    want = ops.mat_mul(a, b, trans_b=True, force=force)
    if m * n < 64 * 64:
        assert torch.equal(ops.mat_mul(a, b, trans_b=True), want)
    if force == 2:
        p = capi.MatMulParams()
        p.dtype, p.m, p.n, p.k, p.trans_b, p.alpha, p.beta, p.batch, p.stride_y = ops.DT[dtype], m, n, k, 1, 1.0, 1.0, 1, m * n
        y = torch.empty(m * n + 1, dtype=dtype, device="cuda")[1:].view(m, n)
        capi.call("mat_mul", p, [a.data_ptr(), b.data_ptr(), 0], [y.data_ptr()], stream=torch.cuda.current_stream().cuda_stream)
        assert torch.equal(y, want)
    assert _ok()


@pytest.mark.parametrize("dtype", HALF)
def test_prefill_sized_and_auto_route(dtype):
    torch.backends.cuda.matmul.allow_tf32 = False
    g = torch.Generator(device="cuda").manual_seed(0)
    a = torch.randn(2048, 4096, device="cuda", generator=g).to(dtype)
    b = (0.02 * torch.randn(4096 + 256, 4096, device="cuda", generator=g)).to(dtype)
    y = ops.mat_mul(a, b, trans_b=True)            # automatic route must pick the tensor-core kernel
    assert _ok()
    want = a.float() @ b.float().T
    torch.testing.assert_close(y.float(), want, atol=2e-2, rtol=1e-2)
    # linearity, a size-independent property: (2A) B^T = 2 (A B^T), exact except where the 16-bit result is subnormal
    y2 = ops.mat_mul((a * 2).to(dtype), b, trans_b=True)
    torch.testing.assert_close(y2.float(), 2 * y.float(), atol=1e-6, rtol=2e-3)
