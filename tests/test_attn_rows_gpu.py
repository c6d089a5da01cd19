"""rg_b200_attention where the tensor-core prefill kernel does not apply: split keys, several query rows per CTA, grouped heads,
every head dimension and type, caches that start off a 16-byte boundary, no workspace.  Tolerances as for the operator's other tests
(fp32 1e-4 / 1e-5 against a fp64 oracle of a sum of up to a thousand terms, 2e-2 / 1e-2 in 16 bits)."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as onp
from refactorgraph_b200 import capi

import _ops as ops

pytestmark = pytest.mark.gpu


def _case(dtype, N, nH, nKV, S, D, past, cap, seed=0):
    rng = np.random.default_rng(seed + N + nH + S + D + past)
    r = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).to(dtype)
    return r(N, nH, S, D), r(N, nKV, S, D), r(N, nKV, S, D), r(N, nKV, cap, D), r(N, nKV, cap, D)


def _check(o, q, k, v, kc, vc, past):
    want, _, _ = onp.attention(*(t.float().numpy() for t in (q, k, v)), past=past, k_cache=kc.float().numpy(), v_cache=vc.float().numpy())
    tol = dict(rtol=1e-4, atol=1e-5) if q.dtype == torch.float32 else dict(rtol=1e-2, atol=2e-2)
    np.testing.assert_allclose(o.float().cpu().numpy(), want, **tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,nH,nKV,S,D,past,cap", [(1, 1, 1, 1, 128, 0, 1), (1, 4, 4, 1, 128, 63, 64), (2, 4, 4, 1, 128, 64, 4000), (1, 8, 2, 1, 128, 1037, 1100),
                                                   (1, 32, 8, 1, 64, 777, 2000), (3, 2, 1, 1, 32, 129, 140), (2, 3, 3, 1, 256, 500, 512), (1, 2, 2, 3, 64, 300, 303),
                                                   (2, 4, 2, 15, 128, 65, 96), (1, 4, 4, 37, 64, 200, 256), (1, 2, 1, 5, 32, 0, 5)])
def test_steps_and_short_prompts(dtype, N, nH, nKV, S, D, past, cap):
    q, k, v, kc, vc = _case(dtype, N, nH, nKV, S, D, past, cap)
    kd, vd = kc.cuda(), vc.cuda()
    o = ops.attention(q.cuda(), k.cuda(), v.cuda(), past=past, k_cache=kd, v_cache=vd)
    _check(o, q, k, v, kc, vc, past)
    assert torch.equal(o, ops.attention(q.cuda(), k.cuda(), v.cuda(), past=past, k_cache=kd, v_cache=vd))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_unaligned_caches_no_workspace_and_workspace_reuse(dtype):
    N, nH, nKV, S, D, past, cap = 2, 8, 4, 1, 128, 500, 640
    q, k, v, kc, vc = _case(dtype, N, nH, nKV, S, D, past, cap)
    p = capi.AttentionParams(ops.DT[dtype], N, nH, nKV, S, D, cap, 1)
    ws = torch.zeros(capi.workspace("attention", p), dtype=torch.uint8, device="cuda")
    assert ws.numel() > 0
    pt, qd, knew, vnew = torch.tensor([past], device="cuda"), q.cuda(), k.cuda(), v.cuda()
    outs = []
    for off, w in ((0, ws), (0, ws), (1, ws), (0, None), (1, None)):
        kd, vd = (torch.zeros(c.numel() + off, dtype=dtype, device="cuda")[off:].copy_(c.flatten()) for c in (kc, vc))
        o = torch.empty_like(qd)
        capi.call("attention", p, [t.data_ptr() for t in (qd, knew, vnew, pt, kd, vd)], [o.data_ptr(), kd.data_ptr(), vd.data_ptr()],
                  ws=w.data_ptr() if w is not None else 0, stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        _check(o, q, k, v, kc, vc, past)
        outs.append(o)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_a_workspace_serves_aligned_and_unaligned_caches(dtype):
    """One workspace for calls whose row blocks differ in number (4 query rows or 2 to a block on aligned caches, 1 on unaligned
    ones): the sums that one call parks must not lie where the other counts arrivals.  Every row of the output is written."""
    N, nH, nKV, S, D, past, cap = 4, 32, 8, 1, 128, 1037, 1100
    q, k, v, kc, vc = _case(dtype, N, nH, nKV, S, D, past, cap)
    p = capi.AttentionParams(ops.DT[dtype], N, nH, nKV, S, D, cap, 1)
    ws = torch.zeros(capi.workspace("attention", p), dtype=torch.uint8, device="cuda")
    pt, qd, knew, vnew = torch.tensor([past], device="cuda"), q.cuda(), k.cuda(), v.cuda()
    for off in (0, 1, 0, 1, 1, 0):
        kd, vd = (torch.zeros(c.numel() + off, dtype=dtype, device="cuda")[off:].copy_(c.flatten()) for c in (kc, vc))
        o = torch.full_like(qd, float("nan"))
        capi.call("attention", p, [t.data_ptr() for t in (qd, knew, vnew, pt, kd, vd)], [o.data_ptr(), kd.data_ptr(), vd.data_ptr()],
                  ws=ws.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        _check(o, q, k, v, kc, vc, past)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,nH,nKV,S,D,past", [(1, 1, 1, 1, 128, 300), (1, 8, 2, 1, 64, 1037), (1, 2, 2, 3, 32, 140), (1, 1, 1, 1, 256, 90)])
@pytest.mark.parametrize("first", [0, 1])
def test_keys_with_a_score_of_minus_infinity_have_no_weight(dtype, N, nH, nKV, S, D, past, first):
    """Whole steps of a warp, whole splits and scattered keys whose scores are -inf, the leading key among them or not."""
    cap = past + S + 7
    q, k, v, kc, vc = _case(dtype, N, nH, nKV, S, D, past, cap)
    q[..., 0] = q[..., 0].abs() + 0.5
    for j in (*range(first, past // 2), *range(past // 2, past, 3)):
        kc[:, :, j, 0] = float("-inf")
    o = ops.attention(q.cuda(), k.cuda(), v.cuda(), past=past, k_cache=kc.cuda(), v_cache=vc.cuda())
    assert bool(o.isfinite().all())
    _check(o, q, k, v, kc, vc, past)


def test_without_a_cache_it_can_be_captured():
    q, k, v, _, _ = _case(torch.float32, 1, 4, 2, 6, 64, 0, 8)
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    want = ops.attention(q, k, v)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        o = ops.attention(q, k, v)
    o.fill_(float("nan"))
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(o, want)


def test_infinite_values_reach_only_the_rows_that_see_them():
    q, k, v, kc, vc = _case(torch.float32, 1, 2, 2, 4, 64, 100, 200)
    vc[0, 0, 150:] = float("inf")    # past the sequence
    v[0, 0, 3, 0] = float("inf")     # the last position: only the last row sees it
    kd, vd = kc.cuda(), vc.cuda()
    o = ops.attention(q.cuda(), k.cuda(), v.cuda(), past=100, k_cache=kd, v_cache=vd).cpu()
    assert o[0, 0, 3, 0].isinf() and o.isfinite().sum() == o.numel() - 1
