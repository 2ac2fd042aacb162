"""The ResNet training step on a B200 against the CPU oracle composed from the per-op fp64 oracle
(tests/resnet_oracle.py), and loss tracking of the tensor-core modes against the CUDA-core fp32 run."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.resnet_oracle import ResNetOracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch


def make_batch(torch, batch, hw, classes, key):
    images = orc.normal((batch, 3, hw, hw), key, "img")
    lab = orc.rng_for(key, "lab").integers(0, classes, batch)
    onehot = np.zeros((batch, classes), dtype=np.float32)
    onehot[np.arange(batch), lab] = 1
    return images, onehot, torch.from_numpy(images).cuda(), torch.from_numpy(onehot).cuda()


@pytest.mark.parametrize("math,tol", [("fp32", 2e-4), ("3xtf32", 2e-4), ("tf32", 5e-2)])
def test_resnet8_step_matches_oracle(torch_cuda, math, tol):
    """ResNet-8 (one block per stage), batch 8, 32x32: loss, logits and every parameter gradient. In fp32 and 3xTF32 mode
    every gradient tensor matches the oracle to 2e-4. TF32 rounding is amplified by the batch-of-8 BatchNorm layers
    (division by the spread of 8 samples), so there each gradient tensor is held to a cosine of 0.995 with the
    oracle's and 5e-2 on loss and logits."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    ctx = Context(0, math=math, sync=True)
    tr = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=32, classes=10)
    oracle = ResNetOracle(1, 32, 10)
    shapes = oracle.param_shapes()
    assert [e["kind"] for e in tr.entries] == [k for k, _ in shapes]
    assert [e["size"] for e in tr.entries] == [int(np.prod(s)) for _, s in shapes]
    host = tr.init_params("r8")
    # perturb gamma / beta so their gradients are exercised away from (1, 0)
    for i, e in enumerate(tr.entries):
        if e["kind"].startswith("bn"):
            host[e["offset"]:e["offset"] + e["size"]] += 0.1 * orc.uniform_pm1((e["size"],), "r8", "bnp", i)
    tr.set_params(host)
    P = [host[e["offset"]:e["offset"] + e["size"]].reshape(s) for e, (_, s) in zip(tr.entries, shapes)]
    images, onehot, dimg, dlab = make_batch(torch, 8, 32, 10, "r8")
    tr.forward(dimg, dlab)
    tr.backward()
    ctx.synchronize()
    loss_ref, G_ref, logits_ref = oracle.run(P, images, onehot)
    assert abs(tr.loss() - loss_ref) <= tol * max(1.0, abs(loss_ref))
    logits = tr.tensor(-1, (8, 10)).cpu().numpy()
    assert orc.max_err_norm(logits, logits_ref) <= tol
    g = tr.grads.cpu().numpy()
    for e, gr in zip(tr.entries, G_ref):
        got = g[e["offset"]:e["offset"] + e["size"]].astype(np.float64)
        want = np.asarray(gr, dtype=np.float64).ravel()
        if math != "tf32":
            assert orc.max_err_norm(got, want) <= tol, (e["kind"], e["dims"])
        else:
            cos = float(got @ want) / max(float(np.linalg.norm(got) * np.linalg.norm(want)), 1e-300)
            assert cos >= 0.995, (e["kind"], e["dims"], cos)
    # one Momentum step: identical to the oracle update applied to the GPU's own gradients
    before_w, before_g = tr.params.cpu().numpy().copy(), g.copy()
    tr.update(0.01 / 8, 0.9, 1e-4)
    ctx.synchronize()
    after = tr.params.cpu().numpy()
    for e in tr.entries:
        sl = slice(e["offset"], e["offset"] + e["size"])
        w, m_, _ = orc.momentum(before_w[sl], before_g[sl], np.zeros(e["size"]), 0.01 / 8, 0.9, 1e-4, e["is_weight"])
        assert orc.max_err_norm(after[sl], w) <= 1e-6
    assert not tr.grads.any()
    tr.close()
    ctx.close()


@pytest.mark.parametrize("math", ["fp32", "3xtf32"])
def test_resnet8_ten_steps_match_oracle(torch_cuda, math):
    """ResNet-8, batch 8: ten consecutive training steps (forward, backward, Momentum update, next forward on the updated
    weights) against the fp64 oracle stepped the same way: every parameter tensor after the tenth step within 2e-4, every
    step's loss within 2e-4."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    steps, lr, beta, l2 = 10, 0.01 / 8, 0.9, 1e-4
    ctx = Context(0, math=math, sync=True)
    tr = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=32, classes=10)
    oracle = ResNetOracle(1, 32, 10)
    shapes = oracle.param_shapes()
    host = tr.init_params("r8x10")
    for i, e in enumerate(tr.entries):
        if e["kind"].startswith("bn"):
            host[e["offset"]:e["offset"] + e["size"]] += 0.1 * orc.uniform_pm1((e["size"],), "r8x10", "bnp", i)
    tr.set_params(host)
    P = [host[e["offset"]:e["offset"] + e["size"]].reshape(s).astype(np.float32) for e, (_, s) in zip(tr.entries, shapes)]
    M = [np.zeros(p.size) for p in P]
    images, onehot, dimg, dlab = make_batch(torch, 8, 32, 10, "r8x10")
    for s in range(steps):
        tr.forward(dimg, dlab)
        tr.backward()
        got_loss = tr.loss()
        tr.update(lr, beta, l2)
        loss_ref, G_ref, _ = oracle.run(P, images, onehot)
        assert abs(got_loss - loss_ref) <= 2e-4 * max(1.0, abs(loss_ref)), s
        for i, e in enumerate(tr.entries):
            w, m_, _ = orc.momentum(P[i].ravel(), np.asarray(G_ref[i]).ravel(), M[i], lr, beta, l2, e["is_weight"])
            P[i], M[i] = np.asarray(w, dtype=np.float32).reshape(P[i].shape), np.asarray(m_, dtype=np.float64)
    ctx.synchronize()
    after = tr.params.cpu().numpy()
    for i, e in enumerate(tr.entries):
        assert orc.max_err_norm(after[e["offset"]:e["offset"] + e["size"]], P[i].ravel()) <= 2e-4, (e["kind"], e["dims"])
    tr.close()
    ctx.close()


def test_bn_groups_reproduce_sharded_gradients(torch_cuda):
    """Data-parallel ranks take BatchNorm statistics on their own shard. A one-GPU run with two BatchNorm groups on a
    batch of 32 must give the gradients two ranks would sum: the executor run separately on each half of the batch
    (what each rank computes; 2e-5) and the fp64 oracle on each half, summed (2e-4; groups of 16 samples keep the
    per-position variances away from the eps = 1e-8 regime in which fp32 rounding is amplified); the loss is the mean
    over all samples."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    B, H = 32, 16
    ctx = Context(0, math="fp32", sync=True)
    full = ResNetTrainer(ctx, batch=B, blocks_per_stage=1, image_hw=32, classes=10)
    half = ResNetTrainer(ctx, batch=H, blocks_per_stage=1, image_hw=32, classes=10)
    host = full.init_params("ghost")
    half.set_params(host)
    full.set_bn_groups(2)
    images, onehot, dimg, dlab = make_batch(torch, B, 32, 10, "ghost")
    full.forward(dimg, dlab)
    full.backward()
    g_full, loss_full = full.grads.cpu().numpy().copy(), full.loss()
    g_sum, loss_sum = np.zeros_like(g_full), 0.0
    oracle = ResNetOracle(1, 32, 10)
    shapes = oracle.param_shapes()
    P = [host[e["offset"]:e["offset"] + e["size"]].reshape(s) for e, (_, s) in zip(full.entries, shapes)]
    G_or = [np.zeros(int(np.prod(s))) for _, s in shapes]
    for h in range(2):
        sl = slice(H * h, H * h + H)
        half.grads.zero_()
        img_h, lab_h = dimg[sl].contiguous(), dlab[sl].contiguous()  # read in place until the backward pass is done
        half.forward(img_h, lab_h)
        half.backward()
        g_sum += half.grads.cpu().numpy()
        loss_sum += half.loss() * H
        _, G_ref, _ = oracle.run(P, images[sl], onehot[sl])
        for i, g in enumerate(G_ref):
            G_or[i] += np.asarray(g, dtype=np.float64).ravel()
    assert abs(loss_full - loss_sum / B) <= 1e-5 * max(1.0, abs(loss_full))
    for i, e in enumerate(full.entries):
        sl = slice(e["offset"], e["offset"] + e["size"])
        assert orc.max_err_norm(g_full[sl], g_sum[sl]) <= 2e-5, (e["kind"], e["dims"])
        assert orc.max_err_norm(g_full[sl], G_or[i]) <= 2e-4, (e["kind"], e["dims"])
    full.close()
    half.close()
    ctx.close()


def test_wgrad_streams_do_not_change_results(torch_cuda):
    """The weight gradients run on streams of their own, concurrently with the rest of the backward pass. On a
    deterministic context (per-CTA partial sums added in a fixed order) gradients after one step and parameters after
    three (eager and as a replayed CUDA graph) are bit-identical for 1 and 3 streams; the inline run (0 streams: its
    kernels split the pixels over more CTAs) and the default context (CTAs add into one accumulator with atomics, in
    whatever order they finish) agree with them to fp32 rounding."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    _, _, dimg, dlab = make_batch(torch, 16, 32, 10, "wstreams")
    results = []
    for n, det in ((1, True), (3, True), (0, True), (2, False)):
        ctx = Context(0, math="tf32", sync=False)
        ctx.set_deterministic(det)
        tr = ResNetTrainer(ctx, batch=16, blocks_per_stage=2, image_hw=32, classes=10)
        tr.set_wgrad_streams(n)
        tr.init_params("wstreams")
        l0 = tr.launches
        tr.forward(dimg, dlab)
        tr.backward()
        ctx.synchronize()
        launches = tr.launches - l0
        g1 = tr.grads.clone()
        tr.update(1e-3)
        tr.step(dimg, dlab, 1e-3)
        g = tr.capture_step(dimg, dlab, 1e-3, warmup=0)
        g.replay()
        ctx.synchronize()
        results.append((g1, tr.params.clone(), launches))
        tr.close()
        ctx.close()
    g1, p, launches = results[1]
    assert torch.equal(g1, results[0][0])
    assert torch.equal(p, results[0][1])
    assert launches == results[0][2]
    for g1, p, launches in results[2:]:
        assert orc.max_err_norm(g1.cpu().numpy(), results[0][0].cpu().numpy()) <= 1e-5
        assert orc.max_err_norm(p.cpu().numpy(), results[0][1].cpu().numpy()) <= 1e-5
    assert results[2][2] == results[0][2]
    assert results[3][2] <= results[0][2]   # the default context adds into the gradient directly: no second kernel


@pytest.mark.parametrize("math", ["tf32", "fp32"])
def test_wide_layers_take_one_route_whatever_the_streams(torch_cuda, math):
    """Filters of more output channels than the weight-gradient kernel's accumulator holds (1x1 to 160): on a default context too the
    gradients of an inline pass and of one on side streams differ by the order of fp32 sums alone (1e-5; TF32 products against
    fp32 ones part by 2e-3)."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import DenseNetTrainer
    _, _, dimg, dlab = make_batch(torch, 16, 16, 10, "wide")
    grads = []
    for n in (0, 2):
        ctx = Context(0, math=math)
        tr = DenseNetTrainer(ctx, batch=16, growth=40, layers=2, image_hw=16)
        tr.set_wgrad_streams(n)
        tr.init_params("wide")
        tr.forward(dimg, dlab)
        tr.backward()
        ctx.synchronize()
        grads.append(tr.grads.cpu().numpy())
        entries = tr.entries
        tr.close()
        ctx.close()
    for e in entries:
        inline, aside = (g[e["offset"]:e["offset"] + e["size"]] for g in grads)
        assert orc.max_err_norm(inline, aside) <= 1e-5, (e["kind"], e["dims"])


def _bn_calls(torch, ctx):
    """BatchNorm + (add +) ReLU by the public calls, which keep nothing between the passes; x and dx may be prefixes of wider tensors."""
    p = lambda t: t.data_ptr()

    def forward(x, wide, gamma, beta, shortcut=None):
        n, P = x.shape[0], gamma.numel()
        y = torch.empty((n,) + tuple(gamma.shape), device="cuda")
        if shortcut is None:
            ctx._check(ctx.lib.cb_bn_fwd_relu_ex(ctx.h, p(x), p(beta), p(gamma), p(y), n, P, wide))
        else:
            ctx._check(ctx.lib.cb_bn_fwd_add_relu(ctx.h, p(x), p(beta), p(gamma), p(shortcut), p(y), n, P))
        return y

    def backward(dy, gamma, x, wide, y, dx, add, dshortcut=None):
        n, P = x.shape[0], gamma.numel()
        dg, db = torch.empty_like(gamma), torch.empty_like(gamma)
        if dshortcut is None:
            ctx._check(ctx.lib.cb_bn_bwd_fused_ex(ctx.h, p(dy), p(gamma), p(x), p(dx), p(dg), p(db), p(y), n, P, wide, wide, add))
        else:
            ctx._check(ctx.lib.cb_bn_bwd_fused_res(ctx.h, p(dy), p(gamma), p(x), p(dx), p(dg), p(db), p(y), p(dshortcut), 0, n, P))
        return dg, db

    return forward, backward


def _model_after_one_pass(torch, cls, batch, key, **shape):
    from crusaderbackend_b200.api import Context
    _, _, dimg, dlab = make_batch(torch, batch, 32, 10, key)
    ctx = Context(0, math="tf32")
    tr = cls(ctx, batch=batch, image_hw=32, **shape)
    host = tr.init_params(key)
    for i, e in enumerate(tr.entries):
        if e["kind"].startswith("bn"):
            host[e["offset"]:e["offset"] + e["size"]] += 0.1 * orc.uniform_pm1((e["size"],), key, "bnp", i)
    tr.set_params(host)
    tr.forward(dimg, dlab)
    tr.backward()
    ctx.synchronize()
    entry = lambda flat, i: flat[tr.entries[i]["offset"]:tr.entries[i]["offset"] + tr.entries[i]["size"]].clone()
    return ctx, tr, lambda i: entry(tr.params, i), lambda i: entry(tr.grads, i)


BN_BATCHES = [16, 17, 24, 32, 33, 48, 64, 65, 96, 128, 129]  # what the passes keep begins at 16 and ends at 128; 1, 2, 4 and 8 samples a thread


@pytest.mark.parametrize("batch", BN_BATCHES)
def test_batchnorm_of_a_residual_model_has_the_bits_of_the_calls(torch_cuda, batch):
    """ResNet-8: every BatchNorm's output, data gradient and parameter gradients, and a projection's shortcut gradient, from the model's
    own inputs of that layer, against cb_bn_fwd_relu / cb_bn_fwd_add_relu and cb_bn_bwd_fused / _res."""
    torch = torch_cuda
    from crusaderbackend_b200.train import ResNetTrainer
    ctx, tr, param, grad = _model_after_one_pass(torch, ResNetTrainer, batch, "bnr", blocks_per_stage=1)
    forward, backward = _bn_calls(torch, ctx)

    def check(x, y, shape, entry, shortcut=None, projected=False):
        dims = (batch,) + shape
        X, Y, dY = tr.tensor(x, dims), tr.tensor(y, dims), tr.tensor(y, dims, grad=True)
        gamma, beta = param(entry).view(shape), param(entry + 1).view(shape)
        R = None if shortcut is None else tr.tensor(shortcut, dims)
        assert torch.equal(forward(X, 0, gamma, beta, R), Y)
        dX, dR = torch.empty_like(X), None if R is None else torch.empty_like(X)
        dg, db = backward(dY, gamma, X, 0, Y, dX, 0, dR)
        assert torch.equal(dX, tr.tensor(x, dims, grad=True))
        assert torch.equal(dg.ravel(), grad(entry)) and torch.equal(db.ravel(), grad(entry + 1))
        if projected:  # (an identity's gradient goes on to take the first convolution's)
            assert torch.equal(dR, tr.tensor(shortcut, dims, grad=True))

    check(1, 2, (16, 32, 32), 1)
    x, entry = 2, 3
    for c, hw in ((16, 32), (32, 16), (64, 8)):
        projected = c > 16
        # filter, gamma, beta, filter, gamma, beta, [filter]; convolution, BatchNorm, convolution, [projection,] BatchNorm + add
        check(x + 1, x + 2, (c, hw, hw), entry + 1)
        check(x + 3, x + 5 if projected else x + 4, (c, hw, hw), entry + 4, x + 4 if projected else x, projected)
        x, entry = (x + 5, entry + 7) if projected else (x + 4, entry + 6)
    tr.close()
    ctx.close()


@pytest.mark.parametrize("batch", BN_BATCHES)
def test_batchnorm_of_a_dense_model_has_the_bits_of_the_calls(torch_cuda, batch):
    """DenseNet, growth 16, two layers a block: inputs that are channel prefixes of a block's buffer, and gradients of that buffer summed over the
    layers in backward order. 32 to 64 channels at 32 x 32, 16 x 16 and 8 x 8: both forms of two batch groups and the narrow one."""
    torch = torch_cuda
    from crusaderbackend_b200.train import DenseNetTrainer
    growth, layers = 16, 2
    ctx, tr, param, grad = _model_after_one_pass(torch, DenseNetTrainer, batch, "bnd", growth=growth, layers=layers)
    forward, backward = _bn_calls(torch, ctx)
    ch, hw, buf, entry = 2 * growth, 32, 1, 1
    nxt = 3  # image 0, buffer 1, its first channels 2
    for block in range(3):
        wide = (batch, ch + layers * growth, hw, hw)
        X, dX, want = tr.tensor(buf, wide), tr.tensor(buf, wide, grad=True), torch.empty(wide, device="cuda")
        stride = wide[1] * hw * hw
        layer_bns = []
        for _ in range(layers):
            layer_bns.append((nxt, ch, entry))                 # on the prefix
            c = 4 * growth                                     # on the 1x1 convolution's output
            dims, shape = (batch, c, hw, hw), (c, hw, hw)
            x, y, dy = tr.tensor(nxt + 1, dims), tr.tensor(nxt + 2, dims), tr.tensor(nxt + 2, dims, grad=True)
            gamma, beta = param(entry + 3).view(shape), param(entry + 4).view(shape)
            assert torch.equal(forward(x, 0, gamma, beta), y)
            dx = torch.empty_like(x)
            dg, db = backward(dy, gamma, x, 0, y, dx, 0)
            assert torch.equal(dx, tr.tensor(nxt + 1, dims, grad=True))
            assert torch.equal(dg.ravel(), grad(entry + 3)) and torch.equal(db.ravel(), grad(entry + 4))
            ch, nxt, entry = ch + growth, nxt + 5, entry + 6   # BN, conv, BN, conv's view, the next prefix
        layer_bns.append((nxt, ch, entry))                     # transition or head, on the whole buffer
        for add, (y_id, c, e) in enumerate(reversed(layer_bns)):
            dims, shape = (batch, c, hw, hw), (c, hw, hw)
            y, dy, gamma, beta = tr.tensor(y_id, dims), tr.tensor(y_id, dims, grad=True), param(e).view(shape), param(e + 1).view(shape)
            assert torch.equal(forward(X, stride, gamma, beta), y)
            dg, db = backward(dy, gamma, X, stride, y, want, 1 if add else 0)
            assert torch.equal(dg.ravel(), grad(e)) and torch.equal(db.ravel(), grad(e + 1))
        assert torch.equal(want, dX)
        if block < 2:  # BN, conv; the next buffer and its first channels
            ch, hw, buf, entry, nxt = ch // 2, hw // 2, nxt + 2, entry + 3, nxt + 4
    tr.close()
    ctx.close()


def test_resnet56_loss_tracks_fp32_run(torch_cuda):
    """ResNet-56, batch 128 of N(0,1) CIFAR-shaped images, uniform labels, He init, momentum 0.9, lr 0.01/128, 200 steps
    on a repeated batch: the loss of the TF32 and of the 3xTF32 tensor-core run stays within 1 % (of the curve's largest
    value) of the CUDA-core fp32 run's, and all three decrease."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    steps = 200
    losses = {}
    _, _, dimg, dlab = make_batch(torch, 128, 32, 10, "r56")
    for math in ("fp32", "tf32", "3xtf32"):
        ctx = Context(0, math=math, sync=False)
        tr = ResNetTrainer(ctx, batch=128, blocks_per_stage=9, image_hw=32, classes=10)
        assert len([e for e in tr.entries if e["kind"] == "conv"]) == 57
        tr.init_params("r56")
        cur = []
        for _ in range(steps):
            tr.step(dimg, dlab, lr=0.01 / 128)
            cur.append(tr.loss())
        ctx.synchronize()
        losses[math] = cur
        tr.close()
        ctx.close()
    a = np.array(losses["fp32"])
    assert np.isfinite(a).all() and a[-1] < a[0]
    for math in ("tf32", "3xtf32"):
        b = np.array(losses[math])
        assert np.isfinite(b).all() and b[-1] < b[0]
        assert np.abs(a - b).max() / np.abs(a).max() <= 0.01, math


@pytest.mark.parametrize("math,tol", [("fp32", 2e-4), ("3xtf32", 2e-4), ("tf32", 5e-2)])
def test_small_densenet_step_matches_oracle(torch_cuda, math, tol):
    """DenseNet-BC with growth 4 and 2 layers per block on 16x16 inputs, batch 16: loss, logits, every gradient
    (fp32: 2e-4 per tensor; TF32: cosine >= 0.98 — fourteen small-batch BatchNorm layers amplify TF32 rounding)."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import DenseNetTrainer
    from tests.model_oracle import densenet_param_shapes, densenet_run
    growth, layers, hw, classes, batch = 4, 2, 16, 10, 16
    ctx = Context(0, math=math, sync=True)
    tr = DenseNetTrainer(ctx, batch=batch, growth=growth, layers=layers, image_hw=hw, classes=classes)
    shapes = densenet_param_shapes(growth, layers, hw, classes)
    assert [e["kind"] for e in tr.entries] == [k for k, _ in shapes]
    assert [e["size"] for e in tr.entries] == [int(np.prod(s)) for _, s in shapes]
    host = tr.init_params("dn")
    for i, e in enumerate(tr.entries):
        if e["kind"].startswith("bn"):
            host[e["offset"]:e["offset"] + e["size"]] += 0.1 * orc.uniform_pm1((e["size"],), "dn", "bnp", i)
    tr.set_params(host)
    P = [host[e["offset"]:e["offset"] + e["size"]].reshape(s) for e, (_, s) in zip(tr.entries, shapes)]
    images, onehot, dimg, dlab = make_batch(torch, batch, hw, classes, "dn")
    tr.forward(dimg, dlab)
    tr.backward()
    ctx.synchronize()
    loss_ref, G_ref, logits_ref = densenet_run(P, images, onehot, growth, layers)
    assert abs(tr.loss() - loss_ref) <= tol * max(1.0, abs(loss_ref))
    assert orc.max_err_norm(tr.tensor(-1, (batch, classes)).cpu().numpy(), logits_ref) <= tol
    g = tr.grads.cpu().numpy()
    for e, gr in zip(tr.entries, G_ref):
        got = g[e["offset"]:e["offset"] + e["size"]].astype(np.float64)
        want = np.asarray(gr, dtype=np.float64).ravel()
        if math != "tf32":
            assert orc.max_err_norm(got, want) <= tol, (e["kind"], e["dims"])
        else:
            cos = float(got @ want) / max(float(np.linalg.norm(got) * np.linalg.norm(want)), 1e-300)
            assert cos >= 0.98, (e["kind"], e["dims"], cos)
    tr.close()
    ctx.close()


def test_densenet_bc_100_forward_backward(torch_cuda):
    """Config 5: DenseNet-BC-100 (k = 12, 3 x 16 bottleneck layers, compression 0.5), batch 64 of 3x32x32 N(0,1)
    images: forward + backward run, the loss is finite and the TF32 loss agrees with the CUDA-core fp32 run."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import DenseNetTrainer
    _, _, dimg, dlab = make_batch(torch, 64, 32, 10, "dn100")
    losses = {}
    for math in ("fp32", "tf32"):
        ctx = Context(0, math=math, sync=False)
        tr = DenseNetTrainer(ctx, batch=64, growth=12, layers=16, image_hw=32, classes=10)
        assert len([e for e in tr.entries if e["kind"] == "conv"]) == 99
        tr.init_params("dn100")
        tr.forward(dimg, dlab)
        tr.backward()
        losses[math] = tr.loss()
        assert torch.isfinite(tr.grads).all()
        tr.close()
        ctx.close()
    assert np.isfinite(losses["fp32"]) and abs(losses["fp32"] - losses["tf32"]) <= 0.01 * abs(losses["fp32"])


@pytest.mark.parametrize("streams", [0, 2])
def test_recorded_passes_match_eager_ones(streams):
    """Forward and backward passes that come back with the same buffers are recorded on their third call: the same bits and
    the same launch count as a context in sync mode, which never records, over alternating batches, a change of math mode,
    a reallocation of the context's scratch and a change of the weight-gradient streams."""
    import torch
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    torch.manual_seed(5)
    batches = [(torch.randn(8, 3, 16, 16, device="cuda"), torch.eye(10, device="cuda")[torch.randint(0, 10, (8,))].contiguous()) for _ in range(2)]
    wide = torch.randn(256, 64, 32, 32, device="cuda")
    W = torch.randn(64, 64, 3, 3, device="cuda")
    results = []
    for sync in (True, False):
        ctx = Context(0, math="tf32", sync=sync)
        ctx.set_deterministic(True)
        tr = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=16)
        tr.set_wgrad_streams(streams)
        tr.init_params("recorded")
        losses, l0 = [], tr.launches
        for i in range(14):
            if i == 8:
                ctx.set_math("3xtf32")
                ctx.conv(W, wide, torch.empty_like(wide), 1, 1, 1, 1)   # grows the scratch the recordings hold
                ctx.set_math("tf32")
            if i == 11:
                tr.set_wgrad_streams(streams)
            tr.step(*batches[i % 2], lr=1e-3)
            losses.append(tr.loss())
        results.append((losses, tr.params.clone(), tr.momentum.clone(), tr.launches - l0))
        tr.close()
        ctx.close()
    (la, pa, ma, na), (lb, pb, mb, nb) = results
    assert la == lb and torch.equal(pa, pb) and torch.equal(ma, mb)
    assert na == nb


def train_on_new_tensors(torch, cls, sync, math="tf32", classes=10, hw=16, steps=9, shift=0, eager_forwards=(),
                         **shape):
    """Steps on other tensors every time, spoilt once the step is queued. shift: floats by which they start past 16 bytes;
    eager_forwards: steps whose forward pass runs in sync mode, which never records, and whose backward pass does not."""
    from crusaderbackend_b200.api import Context
    ctx = Context(0, math=math, sync=sync)
    ctx.set_deterministic(True)
    tr = cls(ctx, batch=8, image_hw=hw, classes=classes, **shape)
    tr.init_params("new tensors")
    gen = torch.Generator(device="cuda").manual_seed(11)
    kept, losses, l0 = [], [], tr.launches
    for i in range(steps):
        images = torch.empty(8 * 3 * hw * hw + 4, device="cuda")[shift:shift + 8 * 3 * hw * hw].view(8, 3, hw, hw)
        labels = torch.empty(8 * classes + 4, device="cuda")[shift:shift + 8 * classes].view(8, classes)
        images.copy_(torch.randn(images.shape, generator=gen, device="cuda"))
        labels.copy_(torch.eye(classes, device="cuda")[torch.randint(0, classes, (8,), generator=gen, device="cuda")])
        kept += [images, labels]     # no address comes back
        if i in eager_forwards:
            ctx.set_sync(True)
        tr.forward(images, labels)
        ctx.set_sync(sync)
        tr.backward()
        tr.update(1e-3)
        losses.append(tr.loss_tensor())
        images.fill_(float("nan"))
        labels.fill_(float("nan"))
    out = [float(x) for x in losses], tr.params.clone(), tr.momentum.clone(), tr.launches - l0
    replays = tr.replays
    tr.close()
    ctx.close()
    return out, replays


def assert_same_run(torch, eager, recorded):
    (la, pa, ma, na), (lb, pb, mb, nb) = eager, recorded
    assert la == lb and torch.equal(pa, pb) and torch.equal(ma, mb) and na == nb


@pytest.mark.parametrize("model", ["resnet", "densenet"])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_recordings_serve_new_input_tensors(torch_cuda, model, shift):
    """A loop that yields new images and labels every step replays its passes from the third step on, with the bits of a
    context that never records, also where the tensors do not start on 16 bytes."""
    from crusaderbackend_b200.train import DenseNetTrainer, ResNetTrainer
    cls, shape = (ResNetTrainer, dict(blocks_per_stage=1)) if model == "resnet" else (DenseNetTrainer, dict(growth=4, layers=2))
    eager, none = train_on_new_tensors(torch_cuda, cls, True, shift=shift, **shape)
    recorded, replays = train_on_new_tensors(torch_cuda, cls, False, shift=shift, **shape)
    assert none == 0 and replays >= 2 * 6
    assert_same_run(torch_cuda, eager, recorded)


def test_backward_after_an_eager_forward_reads_its_images(torch_cuda):
    """The backward pass after an eager forward pass reads the caller's images, not the batch of an earlier replay, although
    it has a recording of its own."""
    from crusaderbackend_b200.train import ResNetTrainer
    eager, _ = train_on_new_tensors(torch_cuda, ResNetTrainer, True, blocks_per_stage=1)
    recorded, replays = train_on_new_tensors(torch_cuda, ResNetTrainer, False, eager_forwards=(5, 6), blocks_per_stage=1)
    assert replays >= 2 * 4
    assert_same_run(torch_cuda, eager, recorded)


@pytest.mark.parametrize("math,hw,classes", [("fp32", 16, 10), ("fp32", 16, 40), ("tf32", 12, 10)])
def test_models_on_the_cuda_cores_are_recorded(torch_cuda, math, hw, classes):
    """fp32 mode and maps the tensor cores do not take have no packed filters that could be stale: their passes replay too."""
    from crusaderbackend_b200.train import ResNetTrainer
    args = dict(math=math, hw=hw, classes=classes, blocks_per_stage=1)
    eager, _ = train_on_new_tensors(torch_cuda, ResNetTrainer, True, **args)
    recorded, replays = train_on_new_tensors(torch_cuda, ResNetTrainer, False, **args)
    assert replays >= 2 * 6
    assert_same_run(torch_cuda, eager, recorded)


def test_dense_layer_of_a_model_sums_in_one_order(torch_cuda):
    """More than 32 classes on 300 features: the forward product would be split over atomic adds if it were a call of its own.
    In a model it takes the launches, and gives the bits, of a deterministic context."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import DenseNetTrainer
    _, _, dimg, _ = make_batch(torch, 8, 8, 40, "dense order")
    dlab = torch.eye(40, device="cuda")[:8].contiguous()
    results = []
    for deterministic in (True, False):
        ctx = Context(0, math="fp32", sync=True)
        ctx.set_deterministic(deterministic)
        tr = DenseNetTrainer(ctx, batch=8, growth=40, layers=4, image_hw=8, classes=40)
        tr.init_params("dense order")
        l0 = tr.launches
        tr.forward(dimg, dlab)
        results.append((tr.launches - l0, tr.tensor(-1, (8, 40)).clone()))
        tr.close()
        ctx.close()
    assert results[0][0] == results[1][0] and torch.equal(results[0][1], results[1][1])


def test_batchnorm_groups_refuse_views(torch_cuda):
    """A dense block's BatchNorm reads a channel prefix of a wider tensor, whose samples are not P apart: groups of samples are
    refused by the forward pass as by the backward pass."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context, CrusaderError
    from crusaderbackend_b200.train import DenseNetTrainer
    _, _, dimg, dlab = make_batch(torch, 8, 16, 10, "groups")
    ctx = Context(0, math="fp32", sync=True)
    tr = DenseNetTrainer(ctx, batch=8, growth=4, layers=2, image_hw=16, classes=10)
    tr.init_params("groups")
    tr.set_bn_groups(2)
    with pytest.raises(CrusaderError, match="views"):
        tr.forward(dimg, dlab)
    tr.set_bn_groups(1)
    tr.forward(dimg, dlab)
    tr.close()
    ctx.close()


def test_recordings_beyond_the_most_that_are_kept(torch_cuda):
    """Six settings make twelve recordings where eight are kept: over two rounds every setting's passes are recorded, evicted and
    recorded again, with the bits and launches of a context that never records."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    _, _, dimg, dlab = make_batch(torch, 8, 16, 10, "evicted")
    results = []
    for sync in (True, False):
        ctx = Context(0, math="tf32", sync=sync)
        ctx.set_deterministic(True)
        tr = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=16)
        tr.init_params("evicted")
        l0, per_setting = tr.launches, []
        for _ in range(2):
            for math in ("tf32", "3xtf32"):
                ctx.set_math(math)
                for groups in (1, 2, 4):
                    tr.set_bn_groups(groups)
                    before = tr.replays
                    for _ in range(6):   # at most: stale filters, larger scratch, twice eager, then replays
                        tr.step(dimg, dlab, lr=1e-4)
                    per_setting.append(tr.replays - before)
        results.append((tr.params.clone(), tr.momentum.clone(), tr.launches - l0, per_setting))
        tr.close()
        ctx.close()
    (pa, ma, na, ra), (pb, mb, nb, rb) = results
    assert torch.equal(pa, pb) and torch.equal(ma, mb) and na == nb
    assert not any(ra) and min(rb) >= 2
    assert rb[6:] == [8] * 6   # second round: everything was evicted, so two eager steps come first again


def test_pass_that_cannot_be_recorded(torch_cuda):
    """A forward pass that fails, and with it its recording, reports its error every time; the model works when its setting is
    put right, and its other recordings are untouched."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context, CrusaderError
    from crusaderbackend_b200.train import ResNetTrainer
    gen = torch.Generator(device="cuda").manual_seed(3)
    dimg = torch.randn(264, 3, 8, 8, generator=gen, device="cuda")   # no batch groups above 256 samples
    dlab = torch.eye(10, device="cuda")[torch.arange(264, device="cuda") % 10].contiguous()
    results = []
    for sync in (True, False):
        ctx = Context(0, math="tf32", sync=sync)
        ctx.set_deterministic(True)
        tr = ResNetTrainer(ctx, batch=264, blocks_per_stage=1, image_hw=8)
        tr.init_params("failing")
        losses = []
        for i in range(10):
            if i in (3, 6):
                tr.set_bn_groups(2)
                for _ in range(4):
                    with pytest.raises(CrusaderError, match="fused kernels"):
                        tr.forward(dimg, dlab)
                tr.set_bn_groups(1)
            tr.step(dimg, dlab, lr=1e-5)
            losses.append(tr.loss())
        results.append((losses, tr.params.clone(), tr.replays))
        tr.close()
        ctx.close()
    (la, pa, _), (lb, pb, replays) = results
    assert la == lb and torch.equal(pa, pb) and replays >= 2 * 6


@pytest.mark.parametrize("math", ["tf32", "3xtf32"])
def test_models_that_share_a_context_with_a_destroyed_one(torch_cuda, math):
    """The packed filters of a destroyed model are forgotten, so that its parameters may be released: by the updates of the
    models that stay, by a graph that was captured while it lived, and by a model that comes after it."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import DenseNetTrainer, ResNetTrainer
    _, _, dimg, dlab = make_batch(torch, 8, 16, 10, "shared")

    def steps(ctx, tr, key, captured=False, between=None):
        tr.init_params(key)
        host = tr.params.cpu().numpy()
        tr.step(dimg, dlab, lr=1e-3)
        graph = tr.capture_step(dimg, dlab, 1e-3) if captured else None
        if captured:
            ctx._check(ctx.lib.cb_freeze_workspace(ctx.h, 0))
        if between:
            between()
        tr.set_params(host)
        for _ in range(4):
            graph.replay() if captured else tr.step(dimg, dlab, lr=1e-3)
        ctx.synchronize()
        return tr.params.clone()

    def fresh():
        ctx = Context(0, math=math)
        ctx.set_deterministic(True)
        return ctx
    want = {}
    for key, captured in (("stays", True), ("after", False)):
        ctx = fresh()
        tr = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=16)
        want[key] = steps(ctx, tr, key, captured)
        alone = ctx.lib.cb_debug_cached_filters(ctx.h)
        tr.close()
        assert ctx.lib.cb_debug_cached_filters(ctx.h) == 0 < alone
        ctx.close()

    ctx = fresh()
    gone = DenseNetTrainer(ctx, batch=8, growth=4, layers=2, image_hw=16)
    steps(ctx, gone, "gone")
    stays = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=16)

    def destroy():   # after the capture, whose table holds the filters of both
        assert ctx.lib.cb_debug_cached_filters(ctx.h) > alone
        gone.close()
        for name in ("params", "grads", "momentum"):
            setattr(gone, name, None)
        assert ctx.lib.cb_debug_cached_filters(ctx.h) == alone
    assert torch.equal(steps(ctx, stays, "stays", True, destroy), want["stays"])
    after = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=16)
    assert torch.equal(steps(ctx, after, "after"), want["after"])
    assert ctx.lib.cb_debug_cached_filters(ctx.h) == 2 * alone
    stays.close()
    after.close()
    ctx.close()


def test_models_that_share_their_parameters(torch_cuda):
    """A second model bound to the first one's buffers, as for a batch of another size: destroying it leaves the first one's packed
    filters, which its recorded passes read, as they are."""
    torch = torch_cuda
    from crusaderbackend_b200.api import Context
    from crusaderbackend_b200.train import ResNetTrainer
    _, _, dimg, dlab = make_batch(torch, 8, 16, 10, "bound twice")
    results = []
    for second in (False, True):
        ctx = Context(0, math="tf32")
        ctx.set_deterministic(True)
        tr = ResNetTrainer(ctx, batch=8, blocks_per_stage=1, image_hw=16)
        tr.init_params("bound twice")
        for i in range(10):
            tr.step(dimg, dlab, lr=1e-3)
            if second and i == 5:
                other = ResNetTrainer(ctx, batch=4, blocks_per_stage=1, image_hw=16)
                other._check(other.lib.cbt_bind(other.h, tr.params.data_ptr(), tr.grads.data_ptr(), tr.momentum.data_ptr()))
                other.forward(dimg[:4], dlab[:4])
                other.close()
        results.append((tr.params.clone(), ctx.lib.cb_debug_cached_filters(ctx.h)))
        assert tr.replays > 0
        tr.close()
        assert ctx.lib.cb_debug_cached_filters(ctx.h) == 0
        ctx.close()
    assert torch.equal(results[0][0], results[1][0])
    assert results[0][1] <= results[1][1]   # another batch may pack some filters in another layout as well
