"""Which convolutions at fp32 accuracy conv_patch_kernel takes, by direction and by whether shares of a contraction may be added up, and the accuracy
of the parameter gradients of dense layers in 3xTF32.

What shows it: a call that adds to its output clears nothing, so two launches are pack_patch_filter and conv_patch_kernel and one is the gathers'.
A plan without shares computes the same on a deterministic context, to the bit; one with shares, added by atomics, cannot over 10^5 outputs.

Tolerances: those of test_conv_patch_gpu.py (2e-6) and of test_gemm_x3_gpu.py (1e-5) for the same arithmetic.
"""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc

from .test_conv_patch_gpu import Epilogue, launches, reference, tensors

pytestmark = pytest.mark.gpu

# forward, data gradient: None (the gathers), or whether the plan has shares; of 148 SMs
ROUTES = {(32, 32, 28, 28, 32, 3, 1, 1): (False, False), (9, 17, 47, 45, 33, 3, 1, 1): (None, False), (20, 40, 33, 29, 70, 3, 1, 0): (None, True),
          (64, 32, 32, 32, 64, 3, 2, 1): (None, False), (24, 64, 61, 47, 31, 3, 2, 1): (None, False), (12, 30, 40, 38, 65, 5, 1, 2): (False, True),
          (40, 64, 40, 40, 64, 1, 1, 0): (False, False), (30, 80, 42, 44, 96, 1, 2, 0): (None, None), (30, 64, 41, 41, 1, 5, 1, 2): (False, None),
          (6, 129, 30, 31, 48, 3, 1, 1): (True, False),
          # a CTA for every SM (75 to 148 of them) and two
          (5, 48, 40, 40, 80, 5, 2, 2): (True, True), (16, 32, 28, 28, 32, 3, 1, 1): (None, True)}


@pytest.mark.parametrize("geo", ROUTES)
def test_routes(geo):
    import torch
    from crusaderbackend_b200.api import Context
    N, IC, H, W_, OC, F, s, p = geo
    W, X, dY = tensors(geo)
    y, dx = reference(W, X, dY, s, p)
    ctx, ep, out = Context(0, math="fp32", sync=True), Epilogue(), {}
    ep.accumulate = 1
    for det in (False, True):
        ctx.set_deterministic(det)
        Y, dX = torch.zeros_like(dY), torch.zeros_like(X)
        torch.cuda.synchronize()
        count = (launches(ctx, lambda: ctx._check(ctx.lib.cb_conv_fwd_ex(ctx.h, W.data_ptr(), X.data_ptr(), Y.data_ptr(), N, IC, H, W_, OC, F, F, s, s, p, p, ctypes.byref(ep)))),
                 launches(ctx, lambda: ctx._check(ctx.lib.cb_conv_dgrad_ex(ctx.h, W.data_ptr(), dY.data_ptr(), dX.data_ptr(), N, IC, H, W_, OC, F, F, s, s, p, p, 1, 0, 0))))
        assert count == tuple(1 if shares is None else 2 for shares in ROUTES[geo])
        assert orc.max_err_norm(Y.cpu().numpy(), y) <= 2e-6
        assert orc.max_err_norm(dX.cpu().numpy(), dx) <= 2e-6
        out[det] = Y, dX
    ctx.close()
    for shares, a, b in zip(ROUTES[geo], out[False], out[True]):
        assert shares is None or torch.equal(a, b) == (not shares)


@pytest.mark.parametrize("outs", [1, 4, 10, 16])
@pytest.mark.parametrize("batch,ins", [(32, 64), (33, 67), (130, 129), (128, 4096)])
def test_parameter_gradients_in_3xtf32(batch, ins, outs):
    import torch
    from crusaderbackend_b200.api import Context
    X, dY = orc.normal((batch, ins), "x3 thin", outs, "X"), orc.normal((batch, outs), "x3 thin", outs, "dY")
    tX, tdY, dW, db = torch.from_numpy(X).cuda(), torch.from_numpy(dY).cuda(), torch.ones(outs, ins, device="cuda"), torch.ones(outs, device="cuda")
    ctx = Context(0, math="3xtf32", sync=True)
    ctx.linearParamGrad(tdY, tX, dW, db)
    ctx.close()
    assert orc.max_err_norm(dW.cpu().numpy(), dY.T.astype(np.float64) @ X + 1) <= 1e-5
    assert orc.max_err_norm(db.cpu().numpy(), dY.astype(np.float64).sum(0) + 1) <= 2e-6
