"""Products at fp32 accuracy on the tensor cores (three bf16 values a factor) against the fp64 CPU oracle.

Tolerance: that of the fp32 CUDA-core kernels, 2e-6 of max|c - c64| / max|c64|. The six products leave out 2^-26 of a term on
average, a chain of 64 k in the tensor core is truncated by four additions (4 x 2^-24 of the chain), the chains are added in fp32.
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

TOL = 2e-6
FORMS = {"NN": (False, False), "NT": (False, True), "TN": (True, False), "TT": (True, True)}


@pytest.fixture(scope="module")
def ctx():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from crusaderbackend_b200.api import Context
    c = Context(0, math="fp32", sync=True)
    yield c
    c.close()


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("M,N,K", [(130, 1030, 130), (129, 65, 2049), (2049, 130, 64), (1000, 17, 1000), (127, 2049, 65), (33, 512, 1024), (1500, 1400, 95)])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_product(ctx, M, N, K, form, pad):
    """Tiles of 128 x 128, 64 and 32 and blocks of 32 k one element below, at and above their sizes; rows on 16 bytes and not;
    contraction whole (deterministic context) or split; overwrite and accumulate; what lies between the rows of C stays."""
    import torch
    tA, tB = FORMS[form]
    A = orc.uniform_pm1((K, M + pad) if tA else (M, K + pad), "split", M, N, K, "A")
    B = orc.uniform_pm1((N, K + pad) if tB else (K, N + pad), "split", M, N, K, "B")
    a, b = A[:, :M if tA else K], B[:, :K if tB else N]
    ref = orc.gemm_f64(np.ascontiguousarray(a), np.ascontiguousarray(b), tA, tB)
    dA, dB = torch.from_numpy(A).cuda()[:, :a.shape[1]], torch.from_numpy(B).cuda()[:, :b.shape[1]]
    whole = torch.full((M, N + 3), 7.0, device="cuda")
    for det in (False, True):
        ctx.set_deterministic(det)
        ctx.gemm(dA, dB, whole[:, :N], transA=tA, transB=tB)
        assert ctx.last_kernel == "umma_fp32"
        assert orc.max_err_norm(whole[:, :N].cpu().numpy(), ref) <= TOL
        ctx.gemm(dA, dB, whole[:, :N], transA=tA, transB=tB, accumulate=True)
        assert orc.max_err_norm(whole[:, :N].cpu().numpy(), 2 * ref) <= TOL
        ctx.set_deterministic(False)
    assert bool((whole[:, N:] == 7).all())


def test_batches_and_dense_layers(ctx):
    import torch
    A, B = orc.uniform_pm1((150, 99), "split", "sA"), orc.uniform_pm1((9, 99, 131), "split", "sB")
    C = torch.zeros(9, 150, 131, device="cuda")
    ctx.sgemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C)
    assert ctx.last_kernel == "umma_fp32"
    assert orc.max_err_norm(C.cpu().numpy(), np.stack([orc.gemm_f64(A, x) for x in B])) <= TOL
    A, B = orc.uniform_pm1((7, 130, 225), "split", "fA"), orc.uniform_pm1((7, 101, 225), "split", "fB")
    C = torch.zeros(130, 101, device="cuda")
    ctx.sgemmNTA(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C)
    assert ctx.last_kernel == "umma_fp32"
    assert orc.max_err_norm(C.cpu().numpy(), sum(orc.gemm_f64(x, y, False, True) for x, y in zip(A, B))) <= TOL
    X, W, b, dY = (orc.normal(s, "split", "lin", i) for i, s in enumerate([(130, 777), (200, 777), (200,), (130, 200)]))
    tX, tW, tb, tdY = (torch.from_numpy(v).cuda() for v in (X, W, b, dY))
    Y, dX, dW, db = torch.zeros(130, 200, device="cuda"), torch.zeros(130, 777, device="cuda"), torch.zeros(200, 777, device="cuda"), torch.zeros(200, device="cuda")
    ctx.linear(tX, tW, tb, Y)
    assert ctx.last_kernel == "umma_fp32"
    assert orc.max_err_norm(Y.cpu().numpy(), X.astype(np.float64) @ W.T + b) <= TOL
    ctx.linearXGrad(tdY, tW, dX)
    ctx.linearParamGrad(tdY, tX, dW, db)
    assert orc.max_err_norm(dX.cpu().numpy(), dY.astype(np.float64) @ W) <= TOL
    assert orc.max_err_norm(dW.cpu().numpy(), dY.T.astype(np.float64) @ X) <= TOL


def test_values_the_pieces_cannot_carry(ctx):
    """Infinities, NaNs and sums that leave the range: such outputs are formed again by fp32 FMAs."""
    import torch
    A, B = orc.uniform_pm1((300, 200), "split", "nA"), orc.uniform_pm1((200, 300), "split", "nB")
    A[3, 5], A[9, 2], A[100, 1], B[7, 11] = np.inf, np.nan, 3.4e38, -np.inf
    C = torch.zeros(300, 300, device="cuda")
    ctx.gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C)
    assert ctx.last_kernel == "umma_fp32"
    got = C.cpu().numpy()
    with np.errstate(invalid="ignore", over="ignore"):
        want = np.zeros((300, 300), np.float32)
        for k in range(200):
            want = want + A[:, k:k + 1] * B[k:k + 1]
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    rows, cols = np.setdiff1d(np.arange(300), [3, 9, 100]), np.setdiff1d(np.arange(300), [11])
    plain = orc.gemm_f64(np.ascontiguousarray(A[rows]), np.ascontiguousarray(B[:, cols]))
    assert orc.max_err_norm(got[np.ix_(rows, cols)], plain) <= TOL
    for sa, sb in [(1e-30, 1.0), (3e38, 1e-3), (1e-25, 1e-10)]:
        A, B = (orc.uniform_pm1((300, 200), "split", "tA") * sa).astype(np.float32), (orc.uniform_pm1((200, 300), "split", "tB") * sb).astype(np.float32)
        ctx.gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C)
        assert orc.max_err_norm(C.cpu().numpy(), orc.gemm_f64(A, B)) <= TOL, (sa, sb)


@pytest.mark.parametrize("geo", [(9, 17, 28, 28, 33, 3, 1, 1), (3, 16, 31, 45, 64, 3, 2, 1), (2, 40, 21, 23, 70, 5, 1, 2), (40, 64, 9, 9, 130, 1, 1, 0),
                                 (2, 16, 45, 44, 20, 17, 1, 8), (33, 20, 13, 13, 100, 3, 3, 1), (5, 130, 14, 14, 31, 3, 1, 1)])
@pytest.mark.parametrize("det", [False, True])
def test_convolution(ctx, geo, det):
    """All passes with odd maps, channels around the tiles, strides whose phases have different taps, and filters on both sides of
    the 15-tap limit of the tap masks; a bias, an accumulating weight gradient, an accumulating data gradient."""
    import torch
    N, IC, H, W_, OC, F, s, p = geo
    OH, OW = orc.conv_out_hw(H, W_, F, F, s, s, p, p)
    W, X, dY = orc.he_normal_filter(OC, IC, F, F, ("split", geo)), orc.normal((N, IC, H, W_), "split", geo, "X"), orc.normal((N, OC, OH, OW), "split", geo, "dY")
    bias, dW0 = orc.normal((OC,), "split", geo, "b"), orc.normal((OC, IC, F, F), "split", geo, "dW0")
    tW, tX, tdY, tb = (torch.from_numpy(v).cuda() for v in (W, X, dY, bias))
    Y, dX, dW = torch.full_like(tdY, float("nan")), torch.full_like(tX, float("nan")), torch.from_numpy(dW0).cuda()
    ctx.set_deterministic(det)
    kern = []
    for call in (lambda: ctx.conv(tW, tX, Y, s, s, p, p, tb), lambda: ctx.convDerive(tW, tdY, dX, s, s, p, p),
                 lambda: ctx.convError(tdY, tX, dW, s, s, p, p)):
        call()
        kern.append(ctx.last_kernel)
    ctx.set_deterministic(False)
    assert kern == ["umma_fp32"] * 3
    assert orc.max_err_norm(Y.cpu().numpy(), orc.conv_fwd(W, X, bias, (s, s), (p, p))) <= TOL
    assert orc.max_err_norm(dX.cpu().numpy(), orc.conv_dgrad(W, dY, X.shape, (s, s), (p, p))) <= TOL
    assert orc.max_err_norm(dW.cpu().numpy(), orc.conv_wgrad(dY, X, W.shape, (s, s), (p, p), dW_init=dW0)) <= TOL


@pytest.mark.parametrize("math,geo,kern", [("3xtf32", (9, 96, 16, 96, 3, 1), ["umma_fp32"] * 3), ("3xtf32", (64, 64, 16, 128, 3, 2), ["umma_fp32", "umma_3xtf32", "umma_fp32"]),
                                           ("3xtf32", (128, 16, 32, 32, 3, 2), ["umma_fp32", "umma_3xtf32", "umma_fp32"]), ("3xtf32", (34, 16, 64, 64, 3, 2), ["umma_3xtf32", "umma_3xtf32", "umma_fp32"]),
                                           ("3xtf32", (34, 16, 64, 32, 3, 2), ["umma_fp32", "umma_3xtf32", "umma_fp32"]), ("tf32", (64, 330, 8, 48, 1, 1), [None, None, "umma_fp32"]),
                                           ("tf32", (4, 128, 16, 128, 3, 1), [None, None, "umma_fp32"])])
def test_passes_of_the_other_modes_that_run_at_fp32_accuracy(math, geo, kern):
    """Wide filters and large stride-2 layers of 3xTF32, weight gradients the TF32 kernel would cut into several launches."""
    import torch
    from crusaderbackend_b200.api import Context
    N, IC, H, OC, F, s = geo
    p = F // 2
    c = Context(0, math=math, sync=True)
    O = (H + 2 * p - F) // s + 1
    W, X, dY = orc.he_normal_filter(OC, IC, F, F, ("other", geo)), orc.normal((N, IC, H, H), "other", geo, "X"), orc.normal((N, OC, O, O), "other", geo, "dY")
    tW, tX, tdY = (torch.from_numpy(v).cuda() for v in (W, X, dY))
    Y, dX, dW = torch.empty_like(tdY), torch.empty_like(tX), torch.zeros_like(tW)
    got = []
    for call in (lambda: c.conv(tW, tX, Y, s, s, p, p), lambda: c.convDerive(tW, tdY, dX, s, s, p, p), lambda: c.convError(tdY, tX, dW, s, s, p, p)):
        call()
        got.append(c.last_kernel)
    c.close()
    assert all(k is None or k == g for k, g in zip(kern, got)), got
    tol = [TOL if g == "umma_fp32" else {"tf32": 2e-3, "3xtf32": 1e-5}[math] for g in got]
    n = min(N, 4)  # a few images of the maps, the whole batch of the weight gradient
    assert orc.max_err_norm(Y[:n].cpu().numpy(), orc.conv_fwd(W, X[:n], None, (s, s), (p, p))) <= tol[0]
    assert orc.max_err_norm(dX[:n].cpu().numpy(), orc.conv_dgrad(W, dY[:n], X[:n].shape, (s, s), (p, p))) <= tol[1]
    ref = torch.nn.grad.conv2d_weight(tX.double(), W.shape, tdY.double(), stride=s, padding=p)
    assert orc.max_err_norm(dW.cpu().numpy(), ref.cpu().numpy()) <= tol[2]


def _elapsed_us(call, reps=3):
    import torch
    call()
    best = float("inf")
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        call()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


def _same_bad_places(got, want, tol=TOL):
    """NaN where the reference has NaN, its infinities where it has them, and its finite values elsewhere."""
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], want[inf].astype(np.float32))
    ok = np.isfinite(want)
    assert not ok.any() or np.abs(got[ok] - want[ok]).max() <= tol * np.abs(want[ok]).max()


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("M,N,K", [(1030, 1030, 95), (300, 260, 1000), (70, 2049, 513), (2049, 40, 256)])
@pytest.mark.parametrize("pad", [1, 4])
def test_products_with_whole_rows_that_are_not_finite(ctx, M, N, K, form, pad):
    """Tiles of every shape in which some outputs, or all, are formed again: an infinity in every row of one factor, NaNs in single
    columns of the other, on both sides of the tiles' edges and in the contraction's first, middle and ragged last block."""
    import torch
    tA, tB = FORMS[form]
    A, B = orc.uniform_pm1((M, K), "again", M, N, K, "A"), orc.uniform_pm1((K, N), "again", M, N, K, "B")
    for i in (0, 31, M - 1):
        A[i, (i * 7) % K] = np.inf if i % 2 else -np.inf
    B[K - 1, N - 1], B[K // 2, 3] = np.nan, np.inf
    every = A.copy()
    every[:, K // 3] = np.inf
    for a in (A, every):
        with np.errstate(invalid="ignore"):
            want = a.astype(np.float64) @ B
        sA, sB = np.ascontiguousarray(a.T if tA else a), np.ascontiguousarray(B.T if tB else B)
        dA, dB = (torch.from_numpy(np.pad(s, ((0, 0), (0, pad)))).cuda()[:, :s.shape[1]] for s in (sA, sB))
        C = torch.full((M, N), 7.0, device="cuda")
        for det in (False, True):
            ctx.set_deterministic(det)
            ctx.gemm(dA, dB, C, transA=tA, transB=tB)
            ctx.set_deterministic(False)
            assert ctx.last_kernel == "umma_fp32"
            _same_bad_places(C.cpu().numpy(), want)


@pytest.mark.parametrize("geo", [(9, 17, 28, 28, 33, 3, 1, 1), (3, 16, 31, 45, 64, 3, 2, 1), (33, 20, 13, 13, 100, 3, 3, 1), (2, 16, 45, 44, 20, 17, 1, 8)])
@pytest.mark.parametrize("det", [False, True])
def test_convolutions_with_values_that_are_not_finite(ctx, geo, det):
    """Infinities in the input and NaNs in the output gradient: all three passes against the same sums as matrix products in fp64."""
    import torch
    N, IC, H, W_, OC, F, s, p = geo
    W = torch.from_numpy(orc.he_normal_filter(OC, IC, F, F, ("bad", geo)))
    X = torch.from_numpy(orc.normal((N, IC, H, W_), "bad", geo, "X"))
    OH, OW = orc.conv_out_hw(H, W_, F, F, s, s, p, p)
    dY = torch.from_numpy(orc.normal((N, OC, OH, OW), "bad", geo, "dY"))
    X[0, 2, 5, 7], X[N - 1, IC - 1, H - 1, W_ - 1] = float("inf"), float("-inf")
    dY[0, 1, 2, 3], dY[N - 1, OC - 1, OH - 1, OW - 1] = float("nan"), float("inf")
    cols = torch.nn.functional.unfold(X.double(), F, padding=p, stride=s)
    fwd = (W.double().reshape(OC, -1) @ cols).reshape(dY.shape)
    wgrad = torch.einsum("nop,nkp->ok", dY.double().reshape(N, OC, -1), cols).reshape(W.shape)
    dgrad = torch.nn.functional.fold(W.double().reshape(OC, -1).T @ dY.double().reshape(N, OC, -1), (H, W_), F, padding=p, stride=s)
    tW, tX, tdY = W.cuda(), X.cuda(), dY.cuda()
    Y, dX, dW = torch.empty_like(tdY), torch.empty_like(tX), torch.zeros_like(tW)
    ctx.set_deterministic(det)
    kern = []
    for call in (lambda: ctx.conv(tW, tX, Y, s, s, p, p), lambda: ctx.convDerive(tW, tdY, dX, s, s, p, p), lambda: ctx.convError(tdY, tX, dW, s, s, p, p)):
        call()
        kern.append(ctx.last_kernel)
    ctx.set_deterministic(False)
    assert kern == ["umma_fp32"] * 3
    for got, want in ((Y, fwd), (dX, dgrad), (dW, wgrad)):
        _same_bad_places(got.cpu().numpy(), want.numpy())


def test_values_that_are_not_finite_cost_a_second_pass(ctx):
    """A program whose training has diverged: a NaN in every output. Forming them again takes a pass over the contraction by fp32 FMAs,
    four times the clocks of a pass on the tensor cores and as many blocks to fetch: bounded by ten times the time of finite values (one
    thread an output, one product after the other, took hundreds)."""
    import torch
    A, B = torch.randn(256, 8192, device="cuda"), torch.randn(8192, 256, device="cuda")
    C = torch.empty(256, 256, device="cuda")
    X, dY, dW = torch.randn(8, 16, 28, 28, device="cuda"), torch.randn(8, 64, 28, 28, device="cuda"), torch.zeros(64, 16, 3, 3, device="cuda")
    for det in (False, True):
        ctx.set_deterministic(det)
        for call, bad in ((lambda: ctx.gemm(A, B, C), A[:, 4000]), (lambda: ctx.convError(dY, X, dW, 1, 1, 1, 1), dY[0, :, 0, 0])):
            finite = _elapsed_us(call)
            assert ctx.last_kernel == "umma_fp32"
            keep = bad.clone()
            bad.fill_(float("nan"))
            again = _elapsed_us(call)
            bad.copy_(keep)
            assert again <= 10 * finite, (det, finite, again)
        ctx.set_deterministic(False)


@pytest.mark.parametrize("terms", [1, 2, 4])
def test_dot_products_of_few_terms(ctx, terms):
    """Rows with one to four values that are not 0 in a contraction of 512 (a diagonal, a mask). Of a term the three products left out
    are at most 2 x 2^-7 2^-16 = 2^-22 (the pieces: 8 bits cut off, so x2 < 2^-7, x3 < 2^-16); a term's largest product is truncated by up to
    2^-23 when it is added, its five small ones together by as much at most, and its chain's sum is rounded by 2^-24 once: (1.5 terms +
    3) 2^-23 of the sum of the terms' magnitudes. A term with a power of two is exact."""
    import torch
    M, N, K = 512, 320, 512
    rng = np.random.default_rng(terms)
    A, B = np.zeros((M, K), np.float32), orc.normal((K, N), "few", terms)
    for i in range(M):
        A[i, rng.choice(K, terms, replace=False)] = rng.standard_normal(terms)
    for a, b in ((A, B), (np.ascontiguousarray(B.T), np.ascontiguousarray(A.T))):
        C = torch.empty(a.shape[0], b.shape[1], device="cuda")
        ctx.gemm(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), C)
        assert ctx.last_kernel == "umma_fp32"
        want, size = a.astype(np.float64) @ b, np.abs(a).astype(np.float64) @ np.abs(b)
        assert (np.abs(C.cpu().numpy() - want) <= (1.5 * terms + 3) * 2.0 ** -23 * size).all()
        if terms == 1:
            two = np.where(a == 0, 0, np.copysign(2.0 ** np.floor(np.log2(np.abs(a) + (a == 0))), a)).astype(np.float32) if a is A else a
            other = b if a is A else np.where(b == 0, 0, np.copysign(2.0 ** np.floor(np.log2(np.abs(b) + (b == 0))), b)).astype(np.float32)
            ctx.gemm(torch.from_numpy(two).cuda(), torch.from_numpy(other).cuda(), C)
            assert np.array_equal(C.cpu().numpy(), two.astype(np.float64) @ other)


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("scale", [1e-30, 8e-34, 4e-34, 1e-35, 5e-38, 1e-40])
@pytest.mark.parametrize("other", [1.0, 1e6])
def test_factors_below_the_range_of_three_pieces(ctx, form, scale, other):
    """Below 2^-110 the third piece is cut off. A factor of that size, all over or in some rows beside ordinary ones, keeps fp32
    accuracy: TOL of the row's largest output, plus the rounding of subnormal sums, 2^-150 an FMA, whether the
    contraction is one CTA's or shared by several, whose sums meet in memory."""
    import torch
    tA, tB = FORMS[form]
    M, N, K = 300, 330, 257
    A = orc.uniform_pm1((M, K), "low", scale, "A")
    A *= np.where((np.arange(M) % 3 == 0) | (M - 1 == np.arange(M)), scale, 1.0 if other == 1.0 else scale)[:, None]
    A = (A * (orc.uniform_pm1((M, K), "low", "mask") > 0)).astype(np.float32)
    B = (orc.uniform_pm1((K, N), "low", scale, "B") * other).astype(np.float32)
    B[:, 17] = 0
    for a, b in ((A, B), (np.ascontiguousarray(B.T), np.ascontiguousarray(A.T))):
        want = a.astype(np.float64) @ b
        dA, dB = torch.from_numpy(np.ascontiguousarray(a.T if tA else a)).cuda(), torch.from_numpy(np.ascontiguousarray(b.T if tB else b)).cuda()
        C = torch.full(want.shape, 7.0, device="cuda")
        for det in (False, True):
            ctx.set_deterministic(det)
            ctx.gemm(dA, dB, C, transA=tA, transB=tB)
            ctx.set_deterministic(False)
            assert ctx.last_kernel == "umma_fp32"
            axis = 1 if a is A else 0
            worst = np.abs(want).max(axis=axis, keepdims=True)
            assert (np.abs(C.cpu().numpy() - want) <= TOL * worst + K * 2.0 ** -150).all()


@pytest.mark.parametrize("geo", [(9, 17, 28, 28, 33, 3, 1, 1), (3, 16, 31, 45, 64, 3, 2, 1), (33, 20, 13, 13, 100, 3, 3, 1), (2, 16, 45, 44, 20, 17, 1, 8)])
def test_convolutions_of_factors_below_the_range_of_three_pieces(ctx, geo):
    """The output gradient of a saturated loss: some channels and images around 1e-36, the others ordinary. Relative to the largest output of
    an image, or of a filter: a sum of K FMAs is a random walk of K roundings by up to 2^-24 of it, 2^-24 sqrt(K / 3) of standard
    deviation, seven of them allowed."""
    import torch
    N, IC, H, W_, OC, F, s, p = geo
    OH, OW = orc.conv_out_hw(H, W_, F, F, s, s, p, p)
    W, X, dY = orc.he_normal_filter(OC, IC, F, F, ("low", geo)), orc.normal((N, IC, H, W_), "low", geo, "X"), orc.normal((N, OC, OH, OW), "low", geo, "dY")
    X[0] *= np.float32(3e-36)
    dY[0] *= np.float32(1e-36)
    dY[:, 1] *= np.float32(2e-36)
    tW, tX, tdY = (torch.from_numpy(v).cuda() for v in (W, X, dY))
    Y, dX, dW = torch.empty_like(tdY), torch.empty_like(tX), torch.zeros_like(tW)
    for det in (False, True):
        ctx.set_deterministic(det)
        dW.zero_()
        for call in (lambda: ctx.conv(tW, tX, Y, s, s, p, p), lambda: ctx.convDerive(tW, tdY, dX, s, s, p, p), lambda: ctx.convError(tdY, tX, dW, s, s, p, p)):
            call()
            assert ctx.last_kernel == "umma_fp32"
        ctx.set_deterministic(False)
        for K, got, want in ((IC * F * F, Y, orc.conv_fwd(W, X, None, (s, s), (p, p))), (OC * F * F, dX, orc.conv_dgrad(W, dY, X.shape, (s, s), (p, p))),
                             (N * OH * OW, dW, orc.conv_wgrad(dY, X, W.shape, (s, s), (p, p)))):
            g, w = (v.reshape(v.shape[0], v.shape[1], -1) if got is not dW else v.reshape(v.shape[0], 1, -1) for v in (got.cpu().numpy(), np.asarray(want, dtype=np.float64)))
            scale = np.abs(w).max(axis=(1, 2), keepdims=True)  # an image's, or an output channel's
            assert (np.abs(g - w) <= 4 * 2.0 ** -24 * K ** 0.5 * scale + K * 2.0 ** -150).all()
