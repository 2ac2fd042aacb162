"""Weight gradients of 3x3 layers on 32-pixel-wide maps, whose stages hold the image rows of several lines once, and the shifted copies of
dY on maps of 8, 16 and 32 pixels, against fp64.

Tolerance: 2e-3 of max|dW - dW64| / max|dW64| in TF32 (10 bits of each factor), 1e-5 in 3xTF32, as in test_conv_gpu.py.
"""
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("math,tol", [("tf32", 2e-3), ("3xtf32", 1e-5)])
@pytest.mark.parametrize("det", [False, True])
@pytest.mark.parametrize("N,IC,H,W,OC", [
    (5, 16, 32, 32, 16),    # four lines a stage
    (3, 48, 32, 32, 12),    # two, two M tiles whose last rows reach past a line's
    (3, 3, 32, 32, 16), (2, 7, 32, 32, 20), (2, 43, 32, 32, 33),  # channels padded to eight
    (4, 16, 30, 32, 16), (3, 16, 33, 32, 16), (3, 24, 5, 32, 40),  # heights that are no multiple of the stage's lines
    (1, 16, 4, 32, 16), (2, 64, 32, 32, 64), (2, 100, 32, 32, 30),  # fewer line groups than CTAs; one line a stage
    (3, 24, 16, 16, 80), (3, 32, 8, 8, 128), (2, 16, 16, 16, 112), (5, 40, 8, 8, 48),  # more rows of dY than the shift warps' first four
])
def test_three_by_three(N, IC, H, W, OC, det, math, tol):
    import torch
    from crusaderbackend_b200.api import Context
    ctx = Context(0, math=math, sync=True)
    ctx.set_deterministic(det)
    X, dY = orc.normal((N, IC, H, W), "rows", N, IC, H, W, OC, "X"), orc.normal((N, OC, H, W), "rows", N, IC, H, W, OC, "dY")
    tX, tdY = torch.from_numpy(X), torch.from_numpy(dY)
    w = torch.zeros(OC, IC, 3, 3, dtype=torch.double, requires_grad=True)
    torch.nn.functional.conv2d(tX.double(), w, padding=1).backward(tdY.double())
    dW = torch.ones(OC, IC, 3, 3, device="cuda")
    ctx.convError(tdY.cuda(), tX.cuda(), dW, 1, 1, 1, 1)
    assert orc.max_err_norm(dW.cpu().numpy() - 1, w.grad.numpy()) <= tol
    if det:
        again = torch.ones_like(dW)
        ctx.convError(tdY.cuda(), tX.cuda(), again, 1, 1, 1, 1)
        assert torch.equal(dW, again)
    ctx.close()
