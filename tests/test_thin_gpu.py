"""Thin products (up to 16 rows or columns) on the CUDA cores against fp64: both operands with k contiguous (thin_rows_kernel), the wide one
with j contiguous (thin_gemm_mn_kernel, with the bias gradient).

Tolerance: 2e-6 of max|c - c64| / max|c64|, that of the fp32 CUDA-core kernels: sums of K products in trees or runs of at most K / 8 FMAs.
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

TOL = 2e-6


@pytest.fixture(scope="module", params=["tf32", "3xtf32", "fp32"])
def ctx(request):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from crusaderbackend_b200.api import Context
    c = Context(0, math=request.param, sync=True)
    yield c
    c.close()


@pytest.mark.parametrize("outs", [1, 4, 5, 8, 9, 10, 16])
@pytest.mark.parametrize("batch,ins", [(32, 64), (33, 67), (130, 129), (129, 128), (37, 1024), (36, 1028), (35, 1025), (40, 2048), (33, 4100), (64, 4096), (101, 1601)])
def test_dense_layer(ctx, outs, batch, ins):
    """Thin extents around the kernels' 4, 8 and 16; rows around a block's four, k around a warp's 128 and a block's 1024, shares of a
    cluster with an empty or a ragged end; rows on 16 bytes and not."""
    import torch
    X, W, b, dY = (orc.normal(s, "thin", outs, batch, ins, i) for i, s in enumerate([(batch, ins), (outs, ins), (outs,), (batch, outs)]))
    tX, tW, tb, tdY = (torch.from_numpy(v).cuda() for v in (X, W, b, dY))
    Y = torch.full((batch, outs), float("nan"), device="cuda")
    ctx.linear(tX, tW, tb, Y)
    assert ctx.last_kernel == "simt_fp32"
    assert orc.max_err_norm(Y.cpu().numpy(), X.astype(np.float64) @ W.T + b) <= TOL
    if ctx.math != "fp32" or outs <= 4 or ins <= 2048:  # the others' shares are added by atomics
        again = torch.empty_like(Y)
        ctx.linear(tX, tW, tb, again)
        assert torch.equal(Y, again)
    if ctx.math == "fp32" or batch <= 64:
        dW, db = torch.ones(outs, ins, device="cuda"), torch.ones(outs, device="cuda")
        ctx.linearParamGrad(tdY, tX, dW, db)
        tol = TOL if ctx.last_kernel == "simt_fp32" else 2e-3
        assert orc.max_err_norm(dW.cpu().numpy(), dY.T.astype(np.float64) @ X + 1) <= tol
        assert orc.max_err_norm(db.cpu().numpy(), dY.astype(np.float64).sum(0) + 1) <= TOL


@pytest.mark.parametrize("det", [False, True])
@pytest.mark.parametrize("thin,wide,K,pad", [(3, 70, 300, 0), (7, 33, 1500, 3), (16, 64, 2000, 0), (16, 64, 2000, 1), (11, 260, 700, 4)])
def test_products_by_either_side(thin, wide, K, pad, det):
    """The thin extent as rows and as columns of C, padded rows, what lies beside C, accumulation."""
    import torch
    from crusaderbackend_b200.api import Context
    ctx = Context(0, math="fp32", sync=True)
    ctx.set_deterministic(det)
    for M, N in ((thin, wide), (wide, thin)):
        A, B = orc.uniform_pm1((M, K + pad), "thin", M, N, K, "A"), orc.uniform_pm1((N, K + pad), "thin", M, N, K, "B")
        ref = orc.gemm_f64(np.ascontiguousarray(A[:, :K]), np.ascontiguousarray(B[:, :K]), False, True)
        whole = torch.full((M, N + 3), 7.0, device="cuda")
        for scale in (1, 2):
            ctx.gemm(torch.from_numpy(A).cuda()[:, :K], torch.from_numpy(B).cuda()[:, :K], whole[:, :N], transB=True, accumulate=scale == 2)
            assert ctx.last_kernel == "simt_fp32"
            assert orc.max_err_norm(whole[:, :N].cpu().numpy(), scale * ref) <= TOL
        assert bool((whole[:, N:] == 7).all())
    ctx.close()
