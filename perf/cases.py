"""Workloads of this library as a user's program issues them: whole training steps, single GEMMs, the three passes of a
convolution layer, a dense layer, and the BatchNorm / ReLU pair, through the public Python entry points.

A case is a dict of plain values; `kind` names the family. Sizes are the ones of this repository's configurations,
benchmark and tests, and generic ones between them.
"""
from __future__ import annotations

import math

import torch

from crusaderbackend_b200.api import Context
from crusaderbackend_b200.train import DenseNetTrainer, ResNetTrainer


def listed():
    return [
        # The headline: one ResNet-56 training step on CIFAR-sized images, recorded once and replayed as a CUDA graph.
        dict(name="resnet56_step_b128", kind="resnet", blocks=9, hw=32, batch=128, math="tf32", graph=True),
        # A small model at a small batch, driven call by call (forward, backward, update) without a graph, as a program
        # does while it is being developed or when its batch size changes: launches and host work count.
        dict(name="resnet8_step_b16_calls", kind="resnet", blocks=1, hw=32, batch=16, math="tf32", graph=False),
        # DenseNet-BC-100 at the batch size its configuration names: many narrow 1x1 and 3x3 layers.
        dict(name="densenet100_step_b64", kind="densenet", growth=12, layers=16, hw=32, batch=64, math="tf32", graph=True),
        # The smallest square product of the configurations.
        dict(name="gemm_512_nn", kind="gemm", form="NN", m=512, n=512, k=512, count=1, math="tf32"),
        # The largest one.
        dict(name="gemm_8192_nt", kind="gemm", form="NT", m=8192, n=8192, k=8192, count=1, math="tf32"),
        # fp32-class accuracy, both operands transposed against the tensor core's preferred order.
        dict(name="gemm_2048_tn_3xtf32", kind="gemm", form="TN", m=2048, n=2048, k=2048, count=1, math="3xtf32"),
        # Extents no tile divides and rows that are not 16-byte aligned: matrices as they come out of user data.
        dict(name="gemm_ragged_nn", kind="gemm", form="NN", m=1000, n=777, k=1501, count=1, math="tf32"),
        # A wide 3x3 layer on 32x32 maps, forward, data gradient and weight gradient.
        dict(name="conv3x3_64_hw32_b128", kind="conv", ic=64, oc=64, hw=32, f=3, s=1, batch=128, math="tf32"),
        # The down-sampling layer between two stages, at fp32-class accuracy.
        dict(name="conv3x3s2_32to64_3xtf32", kind="conv", ic=32, oc=64, hw=32, f=3, s=2, batch=128, math="3xtf32"),
        # A layer on maps whose width no tile divides (28x28 images and the maps they lead to).
        dict(name="conv3x3_32_hw28_b32", kind="conv", ic=32, oc=32, hw=28, f=3, s=1, batch=32, math="tf32"),
        # The classifier of a small network: forward, input gradient and parameter gradients of a dense layer.
        dict(name="dense_4096to10_b128", kind="dense", ins=4096, outs=10, batch=128, math="tf32"),
        # BatchNorm and ReLU as the operand graph calls them one by one, forward and backward, on a first-stage map.
        dict(name="bn_relu_16_hw32_b128", kind="bn", c=16, hw=32, batch=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["resnet", "densenet", "gemm", "gemm", "gemm", "conv", "conv", "conv", "dense", "bn"])
    if kind == "resnet":
        return dict(kind=kind, blocks=rng.randint(1, 9), hw=rng.choice([16, 32]), batch=_log(rng, 16, 128),
                    math=rng.choice(["tf32", "tf32", "3xtf32"]), graph=rng.random() < 0.7)
    if kind == "densenet":
        return dict(kind=kind, growth=12, layers=rng.randint(3, 16), hw=32, batch=_log(rng, 16, 64), math="tf32",
                    graph=rng.random() < 0.7)
    if kind == "gemm":
        prec = rng.choice(["tf32", "tf32", "tf32", "3xtf32", "3xtf32", "fp32"])
        form = rng.choice(["NN", "NT", "TN", "NTA", "batched"])
        top = {"tf32": 8192, "3xtf32": 4096, "fp32": 2048}[prec]
        count = 1
        if form in ("NTA", "batched"):
            top //= 4
            count = _log(rng, 2, 64)
        m, n, k = (_log(rng, 64, top) for _ in range(3))
        if form in ("NN", "NT", "TN") and rng.random() < 0.25:
            n = rng.randint(1, 64)  # thin products of classifier layers
        step = rng.choice([32, 4, 1])  # tile-friendly, 16-byte aligned, any
        m, n, k = (max(step, v // step * step) for v in (m, n, k))
        return dict(kind=kind, form=form, m=m, n=n, k=k, count=count, math=prec)
    if kind == "conv":
        f = rng.choice([3, 3, 3, 1, 5])
        s = 1 if f == 5 else rng.choice([1, 1, 2])
        hw = rng.choice([8, 16, 32, 8, 16, 32, 2 * rng.randint(3, 28), rng.randint(7, 56)])
        ic, oc = _log(rng, 3, 128), _log(rng, 8, 128)
        if rng.random() < 0.6:
            ic, oc = max(16, ic // 16 * 16), max(16, oc // 16 * 16)
        batch = _log(rng, 1, 128)
        while batch > 1 and batch * ic * oc * f * f * hw * hw > 8e8 * s * s:
            batch = batch // 2
        return dict(kind=kind, ic=ic, oc=oc, hw=hw, f=f, s=s, batch=batch,
                    math=rng.choice(["tf32", "tf32", "tf32", "3xtf32", "3xtf32", "fp32"]))
    if kind == "dense":
        return dict(kind=kind, ins=_log(rng, 64, 4096), outs=rng.choice([10, 100, _log(rng, 2, 4096)]), batch=_log(rng, 1, 256),
                    math=rng.choice(["tf32", "3xtf32"]))
    return dict(kind=kind, c=_log(rng, 3, 128), hw=rng.choice([8, 16, 32, rng.randint(5, 40)]), batch=_log(rng, 8, 200))


# ---------------------------------------------------------------------------------------------------- state of a case
class _Trainer:
    """A model, its static input batch and, where the program replays it, the recorded step."""

    def __init__(self, case, seed, rnd, cls, **shape):
        self.ctx = Context(0, math=case["math"])
        self.tr = cls(self.ctx, case["batch"], image_hw=case["hw"], **shape)
        self.tr.init_params(("case", seed))
        self.images = rnd(case["batch"], 3, case["hw"], case["hw"])
        labels = torch.randint(0, 10, (case["batch"],), generator=rnd.gen, device="cuda")
        self.labels = torch.nn.functional.one_hot(labels, 10).float()
        self.lr = 0.01 / case["batch"]
        self.graph = None
        if case["graph"]:
            host = self.tr.params.cpu().numpy()
            self.graph = self.tr.capture_step(self.images, self.labels, self.lr)
            self.tr.set_params(host)  # the warm-up steps of the recording are not part of the run

    def run(self):
        if self.graph is not None:
            self.graph.replay()
        else:
            self.tr.step(self.images, self.labels, self.lr)
        return {"loss": self.tr.loss_tensor(), "params": self.tr.params, "momentum": self.tr.momentum}

    def __del__(self):
        try:
            torch.cuda.synchronize()
            self.graph = None
            self.tr.close()
            self.ctx.close()
        except Exception:
            pass


class _Random:
    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, *shape, std=1.0):
        return torch.randn(shape, generator=self.gen, device="cuda") * std

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.gen, device="cuda") * 2 - 1


def _out_hw(case):
    return (case["hw"] - case["f"] + 2 * (case["f"] // 2)) // case["s"] + 1


def prepare(case, seed):
    rnd = _Random(seed)
    kind = case["kind"]
    if kind == "resnet":
        return dict(case=case, model=_Trainer(case, seed, rnd, ResNetTrainer, blocks_per_stage=case["blocks"]))
    if kind == "densenet":
        return dict(case=case, model=_Trainer(case, seed, rnd, DenseNetTrainer, growth=case["growth"], layers=case["layers"]))
    s = dict(case=case, ctx=Context(0, math=case.get("math", "fp32")))
    if kind == "gemm":
        m, n, k, form, count = case["m"], case["n"], case["k"], case["form"], case["count"]
        lead = (count,) if form in ("NTA", "batched") else ()
        # a batched product shares A, as seblas::sgemm does (one filter matrix against every sample)
        s["A"] = rnd.uniform(k, m) if form == "TN" else rnd.uniform(*(lead if form == "NTA" else ()), m, k)
        s["B"] = rnd.uniform(*lead, n, k) if form in ("NT", "NTA") else rnd.uniform(*lead, k, n)
        s["C"] = torch.zeros((*(lead if form == "batched" else ()), m, n), device="cuda")
    elif kind == "conv":
        ic, oc, hw, f, o = case["ic"], case["oc"], case["hw"], case["f"], _out_hw(case)
        s["W"] = rnd(oc, ic, f, f, std=math.sqrt(2.0 / (ic * f * f)))
        s["X"], s["dY"] = rnd(case["batch"], ic, hw, hw), rnd(case["batch"], oc, o, o)
        s["Y"], s["dX"], s["dW"] = torch.zeros_like(s["dY"]), torch.zeros_like(s["X"]), torch.zeros_like(s["W"])
    elif kind == "dense":
        ins, outs, batch = case["ins"], case["outs"], case["batch"]
        s["W"], s["b"] = rnd(outs, ins, std=math.sqrt(2.0 / ins)), rnd(outs, std=math.sqrt(2.0 / outs))
        s["X"], s["dY"] = rnd(batch, ins), rnd(batch, outs, std=0.1)
        s["Y"], s["dX"] = torch.zeros_like(s["dY"]), torch.zeros_like(s["X"])
        s["dW"], s["db"] = torch.zeros_like(s["W"]), torch.zeros_like(s["b"])
    else:
        shape = (case["batch"], case["c"], case["hw"], case["hw"])
        s["X"], s["dR"] = rnd(*shape) * 2 + 0.5, rnd(*shape)
        s["gamma"], s["beta"] = 1 + 0.1 * rnd(*shape[1:]), 0.1 * rnd(*shape[1:])
        for name in ("Y", "R", "xhat", "dY", "dX"):
            s[name] = torch.zeros(shape, device="cuda")
        for name in ("mean", "var", "dgamma", "dbeta"):
            s[name] = torch.zeros(shape[1:], device="cuda")
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("resnet", "densenet"):
        return s["model"].run()
    ctx = s["ctx"]
    if kind == "gemm":
        call = {"NN": ctx.sgemm, "NT": ctx.sgemmNT, "TN": ctx.sgemmTN, "NTA": ctx.sgemmNTA, "batched": ctx.sgemm}[case["form"]]
        return call(s["A"], s["B"], s["C"])
    if kind == "conv":
        g = (case["s"], case["s"], case["f"] // 2, case["f"] // 2)
        ctx.conv(s["W"], s["X"], s["Y"], *g)
        ctx.convDerive(s["W"], s["dY"], s["dX"], *g)
        ctx.convError(s["dY"], s["X"], s["dW"], *g)  # adds onto dW, as parameter gradients always do
        return {"Y": s["Y"], "dX": s["dX"], "dW": s["dW"]}
    if kind == "dense":
        ctx.linear(s["X"], s["W"], s["b"], s["Y"])
        ctx.linearXGrad(s["dY"], s["W"], s["dX"])
        ctx.linearParamGrad(s["dY"], s["X"], s["dW"], s["db"])
        return {"Y": s["Y"], "dX": s["dX"], "dW": s["dW"], "db": s["db"]}
    ctx.batchNorm(s["X"], s["beta"], s["gamma"], s["mean"], s["var"], s["Y"], s["xhat"])
    ctx.relu(s["Y"], s["R"])
    ctx.reluGradFast(s["Y"], s["dR"], s["dY"])
    ctx.batchNormGrad(s["dY"], s["gamma"], s["X"], s["dX"])
    ctx.batchNormParamGrads(s["dY"], s["xhat"], s["dgamma"], s["dbeta"])
    return {k: s[k] for k in ("mean", "var", "xhat", "Y", "R", "dY", "dX", "dgamma", "dbeta")}


# ---------------------------------------------------------------------------------------------------- work, tolerance
def _model_layers(case):
    """(convolutions as (ic, oc, filter, output width), elements normalised per image, classifier inputs)."""
    hw, convs, norms = case["hw"], [], 0
    if case["kind"] == "resnet":
        convs.append((3, 16, 3, hw))
        norms += 16 * hw * hw
        c = 16
        for stage in range(3):
            oc = 16 << stage
            for b in range(case["blocks"]):
                if stage and b == 0:
                    hw //= 2
                    convs.append((c, oc, 1, hw))
                    norms += oc * hw * hw
                convs += [(c, oc, 3, hw), (oc, oc, 3, hw)]
                norms += 2 * oc * hw * hw
                c = oc
        return convs, norms, c
    k = case["growth"]
    c = 2 * k
    convs.append((3, c, 3, hw))
    for block in range(3):
        for _ in range(case["layers"]):
            convs += [(c, 4 * k, 1, hw), (4 * k, k, 3, hw)]
            norms += (c + 4 * k) * hw * hw
            c += k
        norms += c * hw * hw
        if block < 2:
            convs.append((c, c // 2, 1, hw))
            c, hw = c // 2, hw // 2
    return convs, norms, c


def work(case):
    kind = case["kind"]
    if kind in ("resnet", "densenet"):
        convs, norms, fc = _model_layers(case)
        n = case["batch"]
        params = sum(ic * oc * f * f for ic, oc, f, _ in convs) + 2 * norms + 10 * fc + 10
        macs = n * (sum(ic * oc * f * f * o * o for ic, oc, f, o in convs) + 10 * fc)
        return {"bytes": 4 * (4 * params + n * (3 * case["hw"] ** 2 + 10)), "flops": 6 * macs}
    if kind == "gemm":
        m, n, k, count, form = case["m"], case["n"], case["k"], case["count"], case["form"]
        a, b, c = m * k * (count if form == "NTA" else 1), n * k * count, m * n * (count if form == "batched" else 2 if form == "NTA" else 1)
        return {"bytes": 4 * (a + b + c), "flops": 2 * m * n * k * count}
    if kind == "conv":
        n, o = case["batch"], _out_hw(case)
        x, y, w = n * case["ic"] * case["hw"] ** 2, n * case["oc"] * o * o, case["oc"] * case["ic"] * case["f"] ** 2
        return {"bytes": 4 * (2 * x + 2 * y + 3 * w), "flops": 6 * n * o * o * w}
    if kind == "dense":
        i, o, n = case["ins"], case["outs"], case["batch"]
        return {"bytes": 4 * (3 * i * o + 2 * n * i + 2 * n * o + 3 * o), "flops": 6 * n * i * o}
    p = case["c"] * case["hw"] ** 2
    return {"bytes": 4 * (7 * case["batch"] * p + 6 * p), "flops": 20 * case["batch"] * p}


def tolerance(case):
    kind = case["kind"]
    if kind in ("resnet", "densenet"):
        # a gradient is what the whole chain of layers made of each layer's rounding
        return {"rel": 1e-2 if case["math"] == "tf32" else 1e-4}
    if kind == "bn":
        return {"rel": 2e-5}
    # TF32 keeps 10 bits of each factor; the split form and fp32 sum products that are exact to fp32
    return {"rel": 2e-3 if case["math"] == "tf32" else 1e-5}
