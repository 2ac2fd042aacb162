"""3xTF32 products with one factor in TMEM against fp64.

Tolerance: 1e-5 of max|c - c64| / max|c64|, that of the 3xTF32 kernels. What the split leaves out is 2^-22 of a term; a chain of at most
256 k is 96 additions that truncate (96 x 2^-24 = 5.7e-6 of the chain if all of them lost a whole unit, half that on average).
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

TOL = 1e-5
FORMS = {"NN": (False, False), "NT": (False, True), "TN": (True, False), "TT": (True, True)}


@pytest.fixture(scope="module")
def ctx():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from crusaderbackend_b200.api import Context
    c = Context(0, math="3xtf32", sync=True)
    yield c
    c.close()


def aligned(rows, cols, *key):
    """A matrix whose rows start on 16 bytes."""
    import torch
    whole = orc.uniform_pm1((rows, (cols + 3) // 4 * 4), "x3", rows, cols, *key)
    return np.ascontiguousarray(whole[:, :cols]), torch.from_numpy(whole).cuda()[:, :cols]


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("M,N,K", [(1999, 2050, 65), (2050, 1999, 31), (129, 4097, 1030), (4100, 72, 520), (40, 3000, 2052), (700, 700, 257), (2500, 5000, 36)])
def test_product(ctx, M, N, K, form):
    """Widths of 256, 128, 64, 32 and between them (no halves); one element around tiles and k-blocks; one to four shares, one after
    the other in a CTA too; chunks whole and begun; reproducible and added; overwrite and accumulate; nothing beside C is written."""
    import torch
    tA, tB = FORMS[form]
    a, dA = aligned(*((K, M) if tA else (M, K)), "A")
    b, dB = aligned(*((N, K) if tB else (K, N)), "B")
    ref = orc.gemm_f64(a, b, tA, tB)
    whole = torch.full((M, N + 3), 7.0, device="cuda")
    for det in (False, True):
        ctx.set_deterministic(det)
        ctx.gemm(dA, dB, whole[:, :N], transA=tA, transB=tB)
        assert ctx.last_kernel == "umma_3xtf32"
        assert orc.max_err_norm(whole[:, :N].cpu().numpy(), ref) <= TOL
        first = whole.clone()
        ctx.gemm(dA, dB, whole[:, :N], transA=tA, transB=tB, accumulate=True)
        assert orc.max_err_norm(whole[:, :N].cpu().numpy(), 2 * ref) <= TOL
        if det:
            ctx.gemm(dA, dB, whole[:, :N], transA=tA, transB=tB)
            assert torch.equal(whole, first)
        ctx.set_deterministic(False)
    assert bool((whole[:, N:] == 7).all())


def test_batches_and_dense_layers(ctx):
    import torch
    A, B = orc.uniform_pm1((500, 100), "x3", "sA"), orc.uniform_pm1((9, 100, 516), "x3", "sB")
    C = torch.zeros(9, 500, 516, device="cuda")
    ctx.sgemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C)
    assert orc.max_err_norm(C.cpu().numpy(), np.stack([orc.gemm_f64(A, x) for x in B])) <= TOL
    A, B = orc.uniform_pm1((7, 900, 228), "x3", "fA"), orc.uniform_pm1((7, 1000, 228), "x3", "fB")
    C = torch.zeros(900, 1000, device="cuda")
    ctx.sgemmNTA(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C)
    assert orc.max_err_norm(C.cpu().numpy(), sum(orc.gemm_f64(x, y, False, True) for x, y in zip(A, B))) <= TOL
    X, W, b, dY = (orc.normal(s, "x3", "lin", i) for i, s in enumerate([(1030, 776), (1300, 776), (1300,), (1030, 1300)]))
    tX, tW, tb, tdY = (torch.from_numpy(v).cuda() for v in (X, W, b, dY))
    Y, dX, dW, db = torch.zeros(1030, 1300, device="cuda"), torch.zeros(1030, 776, device="cuda"), torch.zeros(1300, 776, device="cuda"), torch.zeros(1300, device="cuda")
    for det in (False, True):
        ctx.set_deterministic(det)
        ctx.linear(tX, tW, tb, Y)
        assert ctx.last_kernel == "umma_3xtf32"
        assert orc.max_err_norm(Y.cpu().numpy(), X.astype(np.float64) @ W.T + b) <= TOL
        ctx.set_deterministic(False)
    ctx.linearXGrad(tdY, tW, dX)
    ctx.linearParamGrad(tdY, tX, dW, db)
    assert orc.max_err_norm(dX.cpu().numpy(), dY.astype(np.float64) @ W) <= TOL
    assert orc.max_err_norm(dW.cpu().numpy(), dY.T.astype(np.float64) @ X) <= TOL


def test_pointwise_convolution_with_bias_and_relu(ctx):
    """Bias of the other side and ReLU in the epilogue: reproducible only, so always whole."""
    import torch
    X, W, b = orc.normal((6, 64, 30, 32), "x3", "cX"), orc.normal((520, 64, 1, 1), "x3", "cW"), orc.normal((520,), "x3", "cb")
    ref = np.maximum(np.einsum("fc,nchw->nfhw", W[:, :, 0, 0].astype(np.float64), X.astype(np.float64)) + b[None, :, None, None], 0)
    Y = torch.zeros(6, 520, 30, 32, device="cuda")
    ctx.conv(torch.from_numpy(W).cuda(), torch.from_numpy(X).cuda(), Y, biases=torch.from_numpy(b).cuda(), relu=True)
    assert ctx.last_kernel == "umma_3xtf32"
    assert orc.max_err_norm(Y.cpu().numpy(), ref) <= TOL
