"""NaN of any bit pattern in a filter reach every output that reads them, and no other: data gradients of stride 2, whose even and odd columns share
a product of conv_patch_kernel in which a phase may lack a tap."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0x7fc0abe5, 0x7fc00000, 0x7fffffff, -0x3f541b])
@pytest.mark.parametrize("geo, at", [((64, 32, 32, 32, 64, 3, 2, 1), (5, 1, 2, 2)), ((64, 32, 32, 32, 64, 3, 2, 1), (63, 31, 1, 1)), ((24, 64, 61, 47, 31, 3, 2, 1), (7, 0, 0, 2))])
def test_filter_with_a_nan(geo, at, bits):
    import torch
    from crusaderbackend_b200.api import Context
    N, IC, H, W_, OC, F, s, p = geo
    OH, OW = orc.conv_out_hw(H, W_, F, F, s, s, p, p)
    W, dY = [torch.from_numpy(v).cuda() for v in (orc.he_normal_filter(OC, IC, F, F, ("nan", geo)), orc.normal((N, OC, OH, OW), "nan", geo))]
    W.view(torch.int32)[at] = bits
    assert W.isnan().sum() == 1
    dX = torch.zeros((N, IC, H, W_), device="cuda")
    ctx = Context(0, math="fp32", sync=True)
    before = ctx.launches
    ctx.convDerive(W, dY, dX, s, s, p, p)
    assert ctx.launches - before == 2  # pack_patch_filter and conv_patch_kernel
    ctx.close()
    x = torch.zeros((N, IC, H, W_), dtype=torch.float64, requires_grad=True)
    torch.nn.functional.conv2d(x, W.double().cpu(), stride=s, padding=p).backward(dY.double().cpu())
    got, want = dX.cpu().numpy(), x.grad.numpy()
    nan = np.zeros((H, W_), bool)  # the pixels that the tap scatters to
    h, w = s * np.arange(OH) + at[2] - p, s * np.arange(OW) + at[3] - p
    nan[np.ix_(h[(h >= 0) & (h < H)], w[(w >= 0) & (w < W_)])] = True
    assert np.isnan(got[:, at[1]][:, nan]).all()
    nans = np.zeros_like(got, bool)
    nans[:, at[1]] = nan
    assert np.array_equal(np.isnan(got), nans)
    assert orc.max_err_norm(got[~nans], want[~nans]) <= 2e-6
