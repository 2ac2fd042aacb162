"""Thin products around the number of clusters that are resident at a time, where the shares of a contraction halve: clusters of four (32 and 33 of
sixteen thin rows, 64 and 65 of eight) and of eight (13 and 14, 27 and 28), against fp64.

Tolerance: that of test_thin_gpu.py, for the same kernel.
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outs,batch,ins", [(16, 128, 4096), (16, 129, 4096), (10, 133, 3293), (10, 52, 8192), (10, 53, 8192), (16, 64, 8001), (7, 256, 4096), (7, 257, 4100), (5, 108, 8192), (5, 109, 8192)])
def test_dense_layer(outs, batch, ins):
    import torch
    from crusaderbackend_b200.api import Context
    X, W, b = (orc.normal(s, "clusters", outs, batch, ins, i) for i, s in enumerate([(batch, ins), (outs, ins), (outs,)]))
    tX, tW, tb = (torch.from_numpy(v).cuda() for v in (X, W, b))
    Y = torch.full((batch, outs), float("nan"), device="cuda")
    ctx = Context(0, math="tf32", sync=True)
    ctx.linear(tX, tW, tb, Y)
    assert ctx.last_kernel == "simt_fp32"
    again = torch.empty_like(Y)
    ctx.linear(tX, tW, tb, again)
    ctx.close()
    assert torch.equal(Y, again)
    assert orc.max_err_norm(Y.cpu().numpy(), X.astype(np.float64) @ W.T + b) <= 2e-6
