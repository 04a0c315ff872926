"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case goes through the public entry points: the "omarchy_mac_torch" device under torch.nn, torch.optim and autograd, the
Sequential auto-fuse, the torch.compile backend and graphs.capture. A case is a dict of plain values:

  task   train   one optimisation step of one of the package's models (loss, backward, optimizer)
         infer   one forward pass of a trained model
         conv    one convolution layer, forward and backward (grouped = depthwise)
         optim   one optimizer step over a list of parameters
  call   how a training or inference program calls the model: "eager" (nn.Module), "compile" (torch.compile with the package's
         backend) or "graph" (forward and backward recorded once with graphs.capture and replayed; the optimizer is called
         after each replay, as a program with a learning-rate schedule has to)

listed() holds the configurations of the benchmark (bench.py) and its tests; draw() gives further sizes of the same ranges."""

import math
import os
import random

# Programs that use the compile backend beside fused stacks ask for fusion themselves (omt.accelerate): the automatic
# forward pre-hook makes torch.compile trace every further model of a process again.
os.environ.setdefault("OMARCHY_MAC_TORCH_AUTO_FUSE", "0")

import torch
import torch.nn.functional as F

import omarchy_mac_torch_b200 as omt
from omarchy_mac_torch_b200 import graphs, models

MODELS = {
    # name: (constructor, input channels, classes, optimizer)
    "plaincnn": (models.PlainCNN3, 3, 10, "sgd"),
    "separable": (models.SeparableCNN, 1, 10, "adam"),
    "resnet18": (models.ResNet18, 3, 1000, "sgd"),
    "mobilenetv3": (models.MobileNetV3SE, 3, 1000, "adamw"),
    "resnet50": (models.ResNet50, 3, 1000, "sgd"),
}


def listed():
    return [
        # the smallest call: one image through a fused eval stack, where launches and host latency are all there is
        {"name": "plaincnn_infer_b1", "task": "infer", "model": "plaincnn", "call": "eager", "batch": 1, "size": 32},
        # batched scoring with a compiled network (conv + BatchNorm + ReLU epilogues in eval mode)
        {"name": "resnet50_infer_b32", "task": "infer", "model": "resnet50", "call": "compile", "batch": 32, "size": 224},
        # small-network training with the launches recorded as a graph, as the benchmark runs these three
        {"name": "plaincnn_train_b128", "task": "train", "model": "plaincnn", "call": "graph", "batch": 128, "size": 32},
        {"name": "resnet18_train_b32", "task": "train", "model": "resnet18", "call": "graph", "batch": 32, "size": 64},
        {"name": "mobilenetv3_train_b32", "task": "train", "model": "mobilenetv3", "call": "graph", "batch": 32, "size": 224},
        # an ordinary eager loop over a small depthwise-separable network with Adam: 28 -> 14 -> 7 pixels, one input channel
        {"name": "separable_train_b128", "task": "train", "model": "separable", "call": "eager", "batch": 128, "size": 28},
        # the benchmark's headline: ResNet-50, batch 256, compiled
        {"name": "resnet50_train_b256", "task": "train", "model": "resnet50", "call": "compile", "batch": 256, "size": 224},
        # single layers, forward and backward: AlexNet's first layer on images, a mid-network 3x3 layer, a strided layer whose
        # sizes divide nothing, and a large-kernel depthwise layer
        {"name": "conv11x11_s4_b16", "task": "conv", "n": 16, "ci": 3, "co": 64, "ih": 224, "iw": 224, "ks": 11, "stride": 4, "pad": 2, "groups": 1, "bias": True},
        {"name": "conv3x3_256_b128", "task": "conv", "n": 128, "ci": 256, "co": 256, "ih": 28, "iw": 28, "ks": 3, "stride": 1, "pad": 1, "groups": 1, "bias": False},
        {"name": "conv3x3_s2_odd_b13", "task": "conv", "n": 13, "ci": 90, "co": 50, "ih": 57, "iw": 43, "ks": 3, "stride": 2, "pad": 1, "groups": 1, "bias": True},
        {"name": "depthwise5x5_b128", "task": "conv", "n": 128, "ci": 96, "co": 96, "ih": 56, "iw": 56, "ks": 5, "stride": 1, "pad": 2, "groups": 96, "bias": False},
        # the optimizer on its own over a large parameter list
        {"name": "adamw_64m", "task": "optim", "opt": "adamw", "tensors": 160, "numel": 400_000},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["plaincnn", "separable", "resnet18", "mobilenetv3", "resnet50", "infer", "conv", "conv", "conv", "depthwise", "depthwise", "optim"])
    if kind == "plaincnn":
        return {"task": "train", "model": kind, "call": "graph", "batch": _log(rng, 16, 512), "size": 32}
    if kind == "separable":
        return {"task": "train", "model": kind, "call": "eager", "batch": _log(rng, 16, 256), "size": rng.randint(20, 40)}
    if kind == "resnet18":
        return {"task": "train", "model": kind, "call": "graph", "batch": _log(rng, 4, 64), "size": rng.randint(33, 128)}
    if kind == "mobilenetv3":
        return {"task": "train", "model": kind, "call": "graph", "batch": _log(rng, 4, 48), "size": rng.randint(96, 224)}
    if kind == "resnet50":
        return {"task": "train", "model": kind, "call": "compile", "batch": _log(rng, 16, 200), "size": rng.randint(112, 224)}
    if kind == "infer":
        if rng.random() < 0.5:
            return {"task": "infer", "model": "plaincnn", "call": "eager", "batch": _log(rng, 2, 512), "size": 32}
        return {"task": "infer", "model": "resnet50", "call": "compile", "batch": _log(rng, 1, 64), "size": rng.randint(96, 256)}
    if kind == "optim":
        return {"task": "optim", "opt": rng.choice(["sgd", "adam", "adamw"]), "tensors": rng.randint(20, 200), "numel": _log(rng, 1_000, 400_000)}
    while True:
        n, h, w = _log(rng, 1, 128), _log(rng, 7, 224), 0
        w = max(7, min(224, int(h * rng.uniform(0.7, 1.4))))
        if kind == "depthwise":
            c = _log(rng, 16, 576)
            ks, stride = rng.choice([3, 3, 5, 7]), rng.choice([1, 1, 2])
            case = {"task": "conv", "n": n, "ci": c, "co": c, "ih": h, "iw": w, "ks": ks, "stride": stride, "pad": ks // 2, "groups": c, "bias": rng.random() < 0.3}
        else:
            ks, stride = rng.choice([(1, 1), (1, 1), (1, 2), (3, 1), (3, 1), (3, 1), (3, 2), (5, 1), (7, 2), (11, 4)])
            ci = _log(rng, 3, 512) if ks < 7 else rng.choice([1, 3, 4])
            co = _log(rng, 8, 512)
            if rng.random() < 0.7:  # most layers keep their channel counts to multiples of eight
                ci, co = (-(-ci // 8) * 8 if ci > 4 else ci), -(-co // 8) * 8
            if min(h, w) + 2 * (ks // 2) < ks:
                continue
            case = {"task": "conv", "n": n, "ci": ci, "co": co, "ih": h, "iw": w, "ks": ks, "stride": stride, "pad": ks // 2, "groups": 1, "bias": rng.random() < 0.3}
        if n * h * w * max(case["ci"], case["co"] // case["stride"] ** 2) <= 200e6 and work(case)["flops"] <= 6e11 and work(case)["flops"] >= 1e6:
            return case


# ---- what the path cannot do without --------------------------------------------------------------------------------

_shapes = {}


def _conv_work(n, ci, co, ih, iw, oh, ow, ks, groups, passes, input_grad):
    f = 2.0 * n * co * oh * ow * (ci // groups) * ks * ks
    x, y, w = n * ci * ih * iw, n * co * oh * ow, co * (ci // groups) * ks * ks
    flops = f * (1 + (passes > 1) + (passes > 1 and input_grad))
    nbytes = 4.0 * (x + y + w) + (4.0 * (x + y + w) + (4.0 * x if input_grad else 0.0) if passes > 1 else 0.0)
    return flops, nbytes


def _model_layers(name, size):
    """(conv and linear geometries, activation elements of the other layers, parameters) of a model, from its modules on the meta device."""
    key = (name, size)
    if key not in _shapes:
        make, ch, classes, _ = MODELS[name]
        with torch.device("meta"):
            m = make(num_classes=classes).eval()
            convs, hooks = [], []

            def see(mod, args, out):
                x = args[0]
                if isinstance(mod, torch.nn.Linear):
                    convs.append((mod.in_features, mod.out_features, 1, 1, 1, 1, 1, 1))
                else:
                    convs.append((mod.in_channels, mod.out_channels, x.shape[2], x.shape[3], out.shape[2], out.shape[3], mod.kernel_size[0], mod.groups))
            for mod in m.modules():
                if isinstance(mod, (torch.nn.Conv2d, torch.nn.Linear)):
                    hooks.append(mod.register_forward_hook(see))
            m(torch.empty(1, ch, size, size))
            _shapes[key] = (convs, sum(p.numel() for p in m.parameters()))
    return _shapes[key]


def work(case):
    """Each layer's (conv, depthwise, linear) operands read once and results written once per pass over it; elementwise layers
    are counted as fused into their neighbours. Training adds the backward passes and the optimizer's state."""
    if case["task"] == "optim":
        per = {"sgd": 20.0, "adam": 28.0, "adamw": 28.0}[case["opt"]]
        total = case["tensors"] * case["numel"]
        return {"bytes": per * total, "flops": 12.0 * total}
    if case["task"] == "conv":
        oh = (case["ih"] + 2 * case["pad"] - case["ks"]) // case["stride"] + 1
        ow = (case["iw"] + 2 * case["pad"] - case["ks"]) // case["stride"] + 1
        f, b = _conv_work(case["n"], case["ci"], case["co"], case["ih"], case["iw"], oh, ow, case["ks"], case["groups"], 2, True)
        return {"bytes": b, "flops": f}
    convs, params = _model_layers(case["model"], case["size"])
    passes = 2 if case["task"] == "train" else 1
    flops = nbytes = 0.0
    for i, (ci, co, ih, iw, oh, ow, ks, groups) in enumerate(convs):
        f, b = _conv_work(case["batch"], ci, co, ih, iw, oh, ow, ks, groups, passes, i > 0)
        flops, nbytes = flops + f, nbytes + b
    if passes == 2:
        nbytes += params * (16.0 if MODELS[case["model"]][3] == "sgd" else 24.0)
    return {"bytes": nbytes, "flops": flops}


# Four times the distance from the same program in float64 (largest over the outputs of one and of two passes, and over sizes
# of the ranges). Weights after an optimizer step carry the rounding of every layer in front of them: where a rounding moves an
# activation across zero a mask flips, and Adam turns the sign of a vanishing gradient into a whole step.
_TOLERANCE = {
    "plaincnn": (4e-5, 1e-3), "separable": (1e-4, 5e-3), "resnet18": (5e-4, 0.06), "mobilenetv3": (1.2e-3, 0.11), "resnet50": (2.5e-5, 6e-3),
}


def tolerance(case):
    if case["task"] == "optim":
        return {"rel": 1e-6, "max": 1e-5}
    if case["task"] == "conv":  # depthwise: float32 sums; dense: sums of up to 100 000 products
        return {"rel": 2.5e-6, "max": 8e-6} if case["groups"] > 1 else {"rel": 1.2e-4, "max": 4e-4}
    if case["task"] == "infer":
        return {"rel": 4e-5, "max": 1e-4}
    rel, most = _TOLERANCE[case["model"]]
    return {"rel": rel, "max": most}


# ---- prepare --------------------------------------------------------------------------------------------------------


def _flat(tensors):
    """One flat buffer with a 256-byte aligned slot for each tensor, filled from them, and the views of it."""
    offs, n = [], 0
    for t in tensors:
        offs.append(n)
        n += -(-t.numel() // 64) * 64
    flat = torch.zeros(max(n, 1), device=tensors[0].device)
    views = []
    for t, o in zip(tensors, offs):
        v = flat[o:o + t.numel()].view(t.shape)
        v.copy_(t)
        views.append(v)
    return flat, views


def _make_model(name, seed):
    make, ch, classes, opt = MODELS[name]
    torch.manual_seed(seed)
    m = make(num_classes=classes)
    if name == "resnet18":
        models.kaiming_normal_convs(m)
    if name == "resnet50":
        with torch.no_grad():
            for b in m.layers:  # residual branches start small, as large-batch recipes have it
                b.b3.weight.fill_(0.2)
    return m


def _flatten_model(m):
    """Parameters and BatchNorm statistics of `m` as views of two flat buffers (what a checkpoint of the run would hold)."""
    with torch.no_grad():
        ps = list(m.parameters())
        weights, views = _flat([p.data for p in ps])
        for p, v in zip(ps, views):
            p.data = v
        bns = [b for b in m.modules() if isinstance(b, torch.nn.BatchNorm2d)]
        stats, views = _flat([t for b in bns for t in (b.running_mean, b.running_var)])
        for i, b in enumerate(bns):
            b.running_mean, b.running_var = views[2 * i], views[2 * i + 1]
    return weights, stats


def _optimizer(kind, params):
    if kind == "sgd":
        # the first steps of a learning-rate warm-up
        return torch.optim.SGD(params, lr=0.005, momentum=0.9, weight_decay=1e-4)
    if kind == "adam":
        return torch.optim.Adam(params, lr=1e-3)
    return torch.optim.AdamW(params, lr=1e-3, weight_decay=0.01)


def prepare(case, seed):
    D = omt.DEVICE
    g = torch.Generator().manual_seed(seed)
    if case["task"] == "optim":
        r = random.Random(case["tensors"])
        sizes = [max(1, case["numel"] + r.randint(-case["numel"] // 8, case["numel"] // 8)) for _ in range(case["tensors"])]
        total = sum(sizes)
        flats = [torch.randn(total, generator=g) * s for s in (1.0, 1.0, 0.1)] + [torch.rand(total, generator=g) * 0.1]
        w, gr, m, v = (_flat([t.to(D) for t in f.split(sizes)]) for f in flats)
        params = [torch.nn.Parameter(t) for t in w[1]]
        for p, t in zip(params, gr[1]):
            p.grad = t
        opt = _optimizer(case["opt"], params)
        # an optimizer in the middle of a run: its moments exist
        for p, a, b in zip(params, m[1], v[1]):
            opt.state[p] = {"momentum_buffer": a} if case["opt"] == "sgd" else {"step": torch.full((), 10.0, device=D), "exp_avg": a, "exp_avg_sq": b}
        return {"task": "optim", "opt": opt, "out": [w[0], m[0]] + ([] if case["opt"] == "sgd" else [v[0]])}
    if case["task"] == "conv":
        ci, co, ks, groups = case["ci"], case["co"], case["ks"], case["groups"]
        x = torch.randn(case["n"], ci, case["ih"], case["iw"], generator=g)
        if ci > 4:  # inside a network activations are channels-last on this device; images arrive as NCHW
            x = x.contiguous(memory_format=torch.channels_last)
        fan = ci // groups * ks * ks
        w = (torch.rand(co, ci // groups, ks, ks, generator=g) * 2 - 1) / fan ** 0.5
        b = (torch.rand(co, generator=g) * 2 - 1) / fan ** 0.5 if case["bias"] else None
        x, w = x.to(D).requires_grad_(), w.to(D).requires_grad_()
        b = b.to(D).requires_grad_() if b is not None else None
        oh = (case["ih"] + 2 * case["pad"] - ks) // case["stride"] + 1
        ow = (case["iw"] + 2 * case["pad"] - ks) // case["stride"] + 1
        gy = torch.randn(case["n"], co, oh, ow, generator=g).contiguous(memory_format=torch.channels_last).to(D)
        return {"task": "conv", "x": x, "w": w, "b": b, "gy": gy, "stride": case["stride"], "pad": case["pad"], "groups": groups}
    name = case["model"]
    _, ch, classes, opt_kind = MODELS[name]
    model = _make_model(name, seed).to(D)
    x = torch.randn(case["batch"], ch, case["size"], case["size"], generator=g).to(D)
    if case["task"] == "infer":
        with torch.no_grad():
            for b in model.modules():  # statistics of a trained network rather than the initial 0 and 1
                if isinstance(b, torch.nn.BatchNorm2d):
                    b.running_mean.copy_(torch.randn(b.num_features, generator=g) * 0.1)
                    b.running_var.copy_(torch.rand(b.num_features, generator=g) + 0.5)
        model.eval()
        if case["call"] != "compile":
            omt.accelerate(model)
        call = torch.compile(model, backend="omarchy_mac_torch", dynamic=False) if case["call"] == "compile" else model
        state = {"task": "infer", "model": call, "x": x}
        run(state)
        return state
    y = torch.randint(0, classes, (case["batch"],), generator=g).to(D)
    weights, stats = _flatten_model(model)
    kept = weights.clone(), stats.clone()
    opt = _optimizer(opt_kind, model.parameters())
    if case["call"] != "compile":
        omt.accelerate(model)
    call = torch.compile(model, backend="omarchy_mac_torch", dynamic=False) if case["call"] == "compile" else model

    def gradients():
        opt.zero_grad(set_to_none=True)
        loss = F.cross_entropy(call(x), y)
        loss.backward()
        return loss.detach()

    if case["call"] == "graph":
        gradients = graphs.capture(gradients)
    state = {"task": "train", "gradients": gradients, "opt": opt, "weights": weights, "stats": stats, "keep": (model, x, y)}
    run(state)
    # back to the initial weights, so that the first timed step is the first step of the run
    with torch.no_grad():
        weights.copy_(kept[0])
        stats.copy_(kept[1])
        for s in opt.state.values():
            for t in s.values():
                if isinstance(t, torch.Tensor):
                    t.zero_()
    return state


# ---- run ------------------------------------------------------------------------------------------------------------


def run(state):
    if state["task"] == "train":
        loss = state["gradients"]()
        state["opt"].step()
        return {"loss": loss, "weights": state["weights"], "stats": state["stats"]}
    if state["task"] == "infer":
        with torch.no_grad():
            return state["model"](state["x"])
    if state["task"] == "conv":
        x, w, b = state["x"], state["w"], state["b"]
        y = F.conv2d(x, w, b, state["stride"], state["pad"], 1, state["groups"])
        return [y.detach(), *torch.autograd.grad(y, [x, w] + ([b] if b is not None else []), state["gy"])]
    state["opt"].step()
    return state["out"]
