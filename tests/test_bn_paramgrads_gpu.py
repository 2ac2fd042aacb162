"""BatchNorm parameter gradients alone against fp64: batches around the sixteen groups of a block and the eight samples a thread has under way,
positions around a block's 64, on 16 bytes and not.

Tolerance: a position's N products are rounded once, added in 16 runs of at most ceil(N / 16), then run by run: no more than ceil(N / 16) + 16
roundings of 2^-24 of the sum of magnitudes (a single position's sum may cancel, so not of the result).
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
    for got, terms in ((dgamma, tdY.double() * tx.double()), (dbeta, tdY.double())):
        bound = ((N + 15) // 16 + 16) * 2.0 ** -24 * terms.abs().sum(0)
        assert bool(((got.double() - terms.sum(0)).abs() <= bound).all())
    assert bool((whole[:, dY[0].size:] == 5.0).all())
    ctx.close()
