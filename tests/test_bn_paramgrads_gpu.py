"""BatchNorm parameter gradients alone against fp64: batches around the sixteen groups of a block and the eight samples a thread has under way,
positions around a block's 64, on 16 bytes and not.

Tolerance: 2e-6 of max|g - g64| / max|g64|: a position's N products in 16 runs of at most N / 16 additions.
"""
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 15, 16, 17, 127, 128, 129, 250])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 7, 9), (4, 4, 4), (3, 5, 5), (16, 8, 8)])
def test_parameter_gradients(N, shape):
    import torch
    from crusaderbackend_b200.api import Context
    ctx = Context(0, sync=True)
    dY, xhat = orc.normal((N, *shape), "pg", N, shape, "dY"), orc.normal((N, *shape), "pg", N, shape, "xhat")
    tdY, tx = torch.from_numpy(dY).cuda(), torch.from_numpy(xhat).cuda()
    whole = torch.full((2, dY[0].size + 3), 5.0, device="cuda")
    dgamma, dbeta = (w[:dY[0].size].view(shape) for w in whole)
    ctx.batchNormParamGrads(tdY, tx, dgamma, dbeta)
    assert orc.max_err_norm(dgamma.cpu().numpy(), (tdY.double() * tx.double()).sum(0).cpu().numpy()) <= 2e-6
    assert orc.max_err_norm(dbeta.cpu().numpy(), tdY.double().sum(0).cpu().numpy()) <= 2e-6
    assert bool((whole[:, dY[0].size:] == 5.0).all())
    ctx.close()
