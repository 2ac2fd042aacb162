"""Convolutions at fp32 accuracy whose patches are split once for all taps (conv_patch.cu), against the fp64 CPU oracle and against the
gathers that other streams, captures and larger filters use.

Tolerance: 2e-6 of max|y - y64| / max|y64|, as in test_split_gpu.py: the same pieces and products, a chain of 80 k in the tensor core
truncated by five additions in each of three groups (5 x 2^-24 of the chain), the chains added in fp32.
"""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

TOL = 2e-6
# N, IC, H, W, OC, F, stride, padding: one and several chunks of 16 channels with a remainder, columns below, at and above 32 and 64, the last
# tile of the line of positions nearly empty, maps without and with unused rows, even and odd widths at stride 2, 1x1 at stride 2 (sets of
# pixels without a tap), one channel on either side, the most taps
GEOS = [(32, 32, 28, 28, 32, 3, 1, 1), (9, 17, 47, 45, 33, 3, 1, 1), (20, 40, 33, 29, 70, 3, 1, 0), (64, 32, 32, 32, 64, 3, 2, 1), (24, 64, 61, 47, 31, 3, 2, 1),
        (12, 30, 40, 38, 65, 5, 1, 2), (7, 96, 54, 54, 16, 3, 2, 1), (40, 64, 40, 40, 64, 1, 1, 0), (30, 80, 42, 44, 96, 1, 2, 0), (30, 1, 56, 57, 64, 5, 1, 2),
        (30, 64, 41, 41, 1, 5, 1, 2), (6, 129, 30, 31, 48, 3, 1, 1), (16, 16, 50, 50, 16, 5, 1, 1), (25, 16, 40, 40, 40, 4, 2, 1)]
PATCHES = set(GEOS) - {(30, 80, 42, 44, 96, 1, 2, 0)}  # the gathers' own model says less for this one


@pytest.fixture(scope="module")
def ctx():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from crusaderbackend_b200.api import Context
    c = Context(0, math="fp32", sync=True)
    yield c
    c.close()


class Epilogue(ctypes.Structure):
    """cb_epilogue of include/crusader_b200.h."""
    _fields_ = [("bias", ctypes.c_void_p), ("scale", ctypes.c_void_p), ("shift", ctypes.c_void_p), ("per_position", ctypes.c_int), ("relu", ctypes.c_int),
                ("accumulate", ctypes.c_int), ("x_batch_stride", ctypes.c_longlong), ("y_batch_stride", ctypes.c_longlong)]


def launches(ctx, call):
    before = ctx.launches
    call()
    return ctx.launches - before


def tensors(geo):
    import torch
    N, IC, H, W_, OC, F, s, p = geo
    OH, OW = orc.conv_out_hw(H, W_, F, F, s, s, p, p)
    W, X, dY = orc.he_normal_filter(OC, IC, F, F, ("patch", geo)), orc.normal((N, IC, H, W_), "patch", geo, "X"), orc.normal((N, OC, OH, OW), "patch", geo, "dY")
    return [torch.from_numpy(v).cuda() for v in (W, X, dY)]


def reference(W, X, dY, s, p):
    import torch
    x = X.double().cpu().requires_grad_()
    y = torch.nn.functional.conv2d(x, W.double().cpu(), stride=s, padding=p)
    y.backward(dY.double().cpu())
    return y.detach().numpy(), x.grad.numpy()


@pytest.mark.parametrize("geo", GEOS)
def test_passes(ctx, geo):
    """Both passes on the context's own stream (patches: two launches where they pay) and on another (gathers), contraction whole and split."""
    import torch
    W, X, dY = tensors(geo)
    s, p = geo[6], geo[7]
    y, dx = reference(W, X, dY, s, p)
    routes = []
    for det in (False, True):
        ctx.set_deterministic(det)
        Y, dX = torch.full_like(dY, float("nan")), torch.full_like(X, float("nan"))
        routes.append(launches(ctx, lambda: ctx.conv(W, X, Y, s, s, p, p)))
        assert ctx.last_kernel == "umma_fp32"
        routes.append(launches(ctx, lambda: ctx.convDerive(W, dY, dX, s, s, p, p)))
        assert ctx.last_kernel == "umma_fp32"
        assert orc.max_err_norm(Y.cpu().numpy(), y) <= TOL
        assert orc.max_err_norm(dX.cpu().numpy(), dx) <= TOL
        if det:
            again = torch.empty_like(dY)
            ctx.conv(W, X, again, s, s, p, p)
            assert torch.equal(again, Y)
    ctx.set_deterministic(False)
    assert (2 in routes) == (geo in PATCHES)


def test_streams_and_captures_take_the_gathers(ctx):
    """The pieces' scratch belongs to the context's own stream: calls on another one and calls that are captured do without it."""
    import torch
    W, X, dY = tensors(GEOS[0])
    y, dx = reference(W, X, dY, 1, 1)
    Y, dX = torch.empty_like(dY), torch.empty_like(X)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx.lib.cb_set_stream(ctx.h, other.cuda_stream)
    assert launches(ctx, lambda: ctx.convDerive(W, dY, dX, 1, 1, 1, 1)) == 1
    ctx.lib.cb_set_stream(ctx.h, None)
    torch.cuda.synchronize()
    assert orc.max_err_norm(dX.cpu().numpy(), dx) <= TOL
    from crusaderbackend_b200.api import Context
    with torch.cuda.stream(other):
        own = Context(0, math="fp32")
        own.conv(W, X, Y, 1, 1, 1, 1)  # kernels are loaded
        other.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=other):
            assert launches(own, lambda: own.convDerive(W, dY, dX, 1, 1, 1, 1)) == 1
        dX.fill_(float("nan"))
        graph.replay()
        other.synchronize()
        assert orc.max_err_norm(dX.cpu().numpy(), dx) <= TOL
        del graph
        own.close()


def test_epilogues_and_strided_batches(ctx):
    """Bias, ReLU, accumulation, scale and shift by channel and by position, batch strides that are no multiple of anything."""
    import torch
    geo = (12, 30, 40, 38, 65, 5, 1, 2)
    N, IC, H, W_, OC, F, s, p = geo
    W, X, dY = tensors(geo)
    y, dx = reference(W, X, dY, s, p)
    bias = torch.randn(OC, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    Y = torch.empty_like(dY)
    for relu in (False, True):
        assert launches(ctx, lambda: ctx.conv(W, X, Y, s, s, p, p, bias, relu)) == 2
        want = y + bias.cpu().numpy()[None, :, None, None].astype(np.float64)
        assert orc.max_err_norm(Y.cpu().numpy(), np.maximum(want, 0) if relu else want) <= TOL
    wide = torch.full((N, IC * H * W_ + 7), 3.0, device="cuda")
    wide[:, :IC * H * W_] = X.reshape(N, -1)
    out = torch.full((N, OC * H * W_ + 5), 2.0, device="cuda")
    for per_position in (0, 1):
        shape = (OC, H, W_) if per_position else (OC,)
        scale, shift = torch.randn(shape, device="cuda"), torch.randn(shape, device="cuda")
        ep = Epilogue()
        ep.scale, ep.shift, ep.per_position, ep.accumulate = scale.data_ptr(), shift.data_ptr(), per_position, 1
        ep.x_batch_stride, ep.y_batch_stride = wide.stride(0), out.stride(0)
        out.fill_(2.0)
        torch.cuda.synchronize()
        assert launches(ctx, lambda: ctx._check(ctx.lib.cb_conv_fwd_ex(ctx.h, W.data_ptr(), wide.data_ptr(), out.data_ptr(), N, IC, H, W_, OC, F, F, s, s, p, p, ctypes.byref(ep)))) == 2
        view = (lambda t: t.cpu().numpy().astype(np.float64)) if per_position else (lambda t: t.cpu().numpy().astype(np.float64)[:, None, None])
        want = y * view(scale) + view(shift) + 2.0
        assert orc.max_err_norm(out[:, :OC * H * W_].reshape(Y.shape).cpu().numpy(), want) <= TOL
        assert bool((out[:, OC * H * W_:] == 2.0).all())
    grad = torch.full((N, IC * H * W_ + 7), 1.0, device="cuda")
    assert launches(ctx, lambda: ctx._check(ctx.lib.cb_conv_dgrad_ex(ctx.h, W.data_ptr(), dY.data_ptr(), grad.data_ptr(), N, IC, H, W_, OC, F, F, s, s, p, p, 1, 0, grad.stride(0)))) == 2
    assert orc.max_err_norm(grad[:, :IC * H * W_].reshape(X.shape).cpu().numpy(), dx + 1.0) <= TOL
    assert bool((grad[:, IC * H * W_:] == 1.0).all())


@pytest.mark.parametrize("det", [False, True])
@pytest.mark.parametrize("geo", [GEOS[0], (12, 30, 40, 38, 65, 5, 1, 2)])
def test_values_the_pieces_cannot_carry(ctx, geo, det):
    """An infinity, a NaN and factors near the largest and the least magnitudes: what the gathers give, which form such outputs the same way."""
    import torch
    W, X, dY = tensors(geo)
    s, p = geo[6], geo[7]
    other = torch.cuda.Stream()

    def both(W, X):
        got = []
        for stream in (None, other.cuda_stream):
            Y = torch.empty_like(dY)
            torch.cuda.synchronize()
            ctx.lib.cb_set_stream(ctx.h, stream)
            n = launches(ctx, lambda: ctx.conv(W, X, Y, s, s, p, p))
            torch.cuda.synchronize()
            got.append(Y.cpu().numpy())
            if stream is None:
                assert n == 2
        ctx.lib.cb_set_stream(ctx.h, None)
        return got

    ctx.set_deterministic(det)
    Xn, Wn = X.clone(), W.clone()
    Xn[1, 3, 5, 7], Xn[2, 0, 0, 0], Wn[4, 1, 0, 0] = float("inf"), float("nan"), -float("inf")
    a, b = both(Wn, Xn)
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
    assert np.isnan(a[:, 4]).any() and not np.isfinite(a[1]).all()
    fine = np.isfinite(a)
    assert orc.max_err_norm(a[fine], b[fine]) <= 2 * TOL
    # what does not reach a phase of a stride-2 data gradient must not reach its outputs: the same pattern by both routes
    for grad_geo in [(64, 32, 32, 32, 64, 3, 2, 1), (24, 64, 61, 47, 31, 3, 2, 1)]:
        gW, gX, gdY = tensors(grad_geo)
        gdY[1, 2, 3, 4], gdY[0, 0, 0, 0], gW[5, 1, 2, 2] = float("inf"), float("nan"), float("inf")
        ref = []
        for stream in (None, other.cuda_stream):
            dX = torch.empty_like(gX)
            torch.cuda.synchronize()
            ctx.lib.cb_set_stream(ctx.h, stream)
            n = launches(ctx, lambda: ctx.convDerive(gW, gdY, dX, 2, 2, 1, 1))
            assert n == (2 if stream is None else n)
            torch.cuda.synchronize()
            ref.append(dX.cpu().numpy())
        ctx.lib.cb_set_stream(ctx.h, None)
        a, b = ref
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
        fine = np.isfinite(a)
        assert 0.5 < fine.mean() < 1 and orc.max_err_norm(a[fine], b[fine]) <= 2 * TOL
    for scale in (1e-36, 1e-30, 1e37):
        a, b = both(W, X * scale)
        y, _ = reference(W, X * scale, dY, s, p)
        assert orc.max_err_norm(a, y) <= TOL, scale
    ctx.set_deterministic(False)
