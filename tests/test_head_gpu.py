"""The classifier head's forward kernel against fp64: planes around a lane's one, four and five positions, channels around a warp's four and a
round of all warps, classes up to a warp's lanes; blocks of sixteen and of thirty-two warps.

Tolerance: a plane's sum has ceil(HW / 32) + 5 roundings and a division, a logit ceil(C / 32) + 5 and the bias, each of 2^-24 of what is summed in
magnitude; a softmax moves by at most twice what its logits do, and expf, the sum of 32 and the quotient add less than 16 roundings.
"""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,C,HW,M", [(1, 1, 1, 1), (3, 4, 31, 10), (2, 5, 33, 32), (5, 64, 64, 10), (3, 33, 127, 17), (2, 63, 128, 10), (2, 65, 129, 10), (2, 256, 196, 10),
                                      (4, 17, 1000, 3), (2, 600, 16, 5), (130, 131, 49, 10)])
def test_forward(N, C, HW, M):
    import torch
    from crusaderbackend_b200.api import Context
    X, W, b = (orc.normal(s, "head", N, C, HW, M, i) for i, s in enumerate([(N, C, HW), (M, C), (M,)]))
    labels = np.eye(M, dtype=np.float32)[np.arange(N) % M]
    dev = [torch.from_numpy(v).cuda() for v in (X, W, b, labels)]
    out = [torch.full(s, float("nan"), device="cuda") for s in ((N, C), (N, M), (N, M), (N, M), (N,))]
    ctx = Context(0, sync=True)
    ctx._check(ctx.lib.cb_head_fwd(ctx.h, *[t.data_ptr() for t in dev + out], N, C, HW, M))
    ctx.close()
    pooled, logits, probs, dlogits, loss = (t.cpu().numpy().astype(np.float64) for t in out)
    eps, X, W, b = 2.0 ** -24, X.astype(np.float64), W.astype(np.float64), b.astype(np.float64)
    mean, size, first, second = X.mean(2), np.abs(X).mean(2), -(-HW // 32) + 6, -(-C // 32) + 6
    assert (np.abs(pooled - mean) <= first * eps * size).all()
    want = mean @ W.T + b
    off = (first + second) * eps * (size @ np.abs(W).T + np.abs(b))
    assert (np.abs(logits - want) <= off).all()
    e = np.exp(want - want.max(1, keepdims=True))
    p = e / (e.sum(1, keepdims=True) + 1e-10)
    off = 2 * off.max(1, keepdims=True) + 16 * eps
    assert (np.abs(probs - p) <= off).all()
    assert (np.abs(dlogits - (p - labels)) <= off + eps).all()
    ce = -(np.log(p + 1e-10) * labels).sum(1)
    assert (np.abs(loss - ce) <= 2 * (off / p * labels).max(1) + 4 * eps * (1 + np.abs(ce))).all()
