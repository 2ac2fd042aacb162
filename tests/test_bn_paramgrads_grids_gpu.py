"""BatchNorm parameter gradients in grids below and above two blocks an SM, where positions that are read one by one change from eight samples of a
thread to four, against fp64. Tolerance: as in test_bn_paramgrads_gpu.py."""
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [3, 64, 65, 129])
@pytest.mark.parametrize("P", [18942, 18944, 18945, 18948])
def test_parameter_gradients(N, P):
    import torch
    from crusaderbackend_b200.api import Context
    ctx = Context(0, sync=True)
    dY, xhat = (torch.from_numpy(orc.normal((N, P, 1, 1), "pg grid", N, P, i)).cuda() for i in range(2))
    whole = torch.full((2, P + 8), 5.0, device="cuda")
    dgamma, dbeta = (w[:P].view(P, 1, 1) for w in whole)
    ctx.batchNormParamGrads(dY, xhat, dgamma, dbeta)
    for got, terms in ((dgamma, dY.double() * xhat.double()), (dbeta, dY.double())):
        bound = ((N + 15) // 16 + 16) * 2.0 ** -24 * terms.abs().sum(0)
        assert bool(((got.double() - terms.sum(0)).abs() <= bound).all())
    assert bool((whole[:, P:] == 5.0).all())
    ctx.close()
