"""What this framework is asked to do in earnest on one GPU, as cases that can be timed.

Five kinds of work, each through the entry points a program calls:

* ``train``      one step of an image classifier (``TrainStep``): ResNet-50 at batch 256 captured in a CUDA graph is the
                 headline benchmark; ResNet-32 at batch 128 is the CIFAR-10 configuration; without a graph (the default
                 of the training program, and the only form in which a wrapped optimizer such as LARS runs) the host's
                 share of a step counts too
* ``sequence``   one step of the 2-layer LSTM classifier over 2048-d frame features; the length changes from batch to
                 batch (30 to 1800 frames), so a step is never captured
* ``evaluate``   a ResNet's inference forward pass, from one image to a validation batch
* ``allreduce``  post + wait of a partial allreduce by itself, 4 KB to 256 MB, fp32 and bf16, even and ragged counts
* ``dense``      a dense layer forward and backward at the sizes of the GEMM benchmark (rows x outputs x inputs)
"""
import math

import torch

import eagersgd_b200 as es
from eagersgd_b200.models.lstm import LSTMClassifier
from eagersgd_b200.models.resnet import IMAGENET_BLOCKS, cifar_resnet, imagenet_resnet
from eagersgd_b200.ops import functional as ops
from eagersgd_b200.optim.lars import LARS
from eagersgd_b200.train.step import TrainStep, prepare_model

FRAME_FEATURES = 2048
VIDEO_CLASSES = 101


def listed():
    return [
        # ImageNet training as the headline benchmark runs it
        _train("train resnet50 b256 graph", "imagenet", 50, 256, 224, "solo", "sgd", True),
        # the large-batch recipe: LARS around a smaller per-GPU batch; a wrapped optimizer is never captured
        _train("train resnet50 b64 lars", "imagenet", 50, 64, 224, "solo", "lars", False),
        # the CIFAR-10 benchmark configuration
        _train("train resnet32 b128 graph", "cifar10", 32, 128, 32, "majority", "sgd", True),
        # the CIFAR-10 recipe as the training program runs it by default: no graph; a batch that is no power of two
        _train("train resnet44 b100", "cifar10", 44, 100, 32, "solo", "sgd", False),
        # short, usual and long clips of the video configuration
        _sequence("sequence 37 frames", 37, 16, 2048),
        _sequence("sequence 331 frames", 331, 16, 2048),
        _sequence("sequence 1203 frames", 1203, 16, 2048),
        # a single request, and the ragged batch at the end of a validation pass
        _evaluate("evaluate resnet50 b1", "imagenet", 50, 1, 224),
        _evaluate("evaluate resnet50 b125", "imagenet", 50, 125, 224),
        # the smallest message, where latency is all there is, and one ~25 MB gradient bucket that is not a multiple of 8
        _allreduce("allreduce fp32 1024", "float32", 1024, "solo"),
        _allreduce("allreduce bf16 13107197", "bfloat16", 13107197, "solo"),
        # a size from the GEMM benchmark whose output width needs padding
        _dense("dense 5124x9124x1760", 5124, 9124, 1760, True),
    ]


def _train(name, dataset, size, batch, res, mode, optimizer, graph):
    return {"name": name, "kind": "train", "dataset": dataset, "size": size, "batch": batch, "res": res, "mode": mode,
            "optimizer": optimizer, "graph": graph}


def _sequence(name, frames, batch, hidden):
    return {"name": name, "kind": "sequence", "frames": frames, "batch": batch, "hidden": hidden}


def _evaluate(name, dataset, size, batch, res):
    return {"name": name, "kind": "evaluate", "dataset": dataset, "size": size, "batch": batch, "res": res}


def _allreduce(name, dtype, count, mode):
    return {"name": name, "kind": "allreduce", "dtype": dtype, "count": count, "mode": mode}


def _dense(name, rows, outputs, inputs, bias):
    return {"name": name, "kind": "dense", "rows": rows, "outputs": outputs, "inputs": inputs, "bias": bias}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "sequence", "sequence", "evaluate", "evaluate", "allreduce", "allreduce",
                       "dense"])
    if kind in ("train", "evaluate"):
        if rng.random() < 0.6:
            dataset, size, res = "imagenet", rng.choice([18, 34, 50]), rng.choice([128, 160, 192, 224])
            batch = _log_int(rng, 8 if kind == "train" else 1, 256)
        else:
            dataset, size, res = "cifar10", rng.choice([20, 32, 44, 56]), 32
            batch = _log_int(rng, 32 if kind == "train" else 1, 512)
        if kind == "evaluate":
            case = _evaluate("", dataset, size, batch, res)
        else:
            optimizer = "lars" if rng.random() < 0.2 else "sgd"
            case = _train("", dataset, size, batch, res, rng.choice(["solo", "majority", "sync"]), optimizer,
                          optimizer == "sgd" and rng.random() < 0.6)
    elif kind == "sequence":
        batch = rng.choice([8, 16, 24, 32])
        case = _sequence("", _log_int(rng, 30, 1203 * 16 // max(batch, 16)), batch, rng.choice([256, 512, 1024, 2048]))
    elif kind == "allreduce":
        dtype = rng.choice(["float32", "bfloat16"])
        count = _log_int(rng, 4 << 10, 256 << 20) // (4 if dtype == "float32" else 2)
        case = _allreduce("", dtype, count, rng.choice(["solo", "majority", "sync"]))
    else:
        case = _dense("", _log_int(rng, 16, 8192), _log_int(rng, 10, 9124), 8 * _log_int(rng, 64, 512), rng.random() < 0.5)
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------------------- preparation
def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + salt) % (1 << 62))


def _randn(seed, salt, *shape):
    return torch.randn(*shape, device="cuda", generator=_generator(seed, salt))


def _classes(case):
    return 1000 if case["dataset"] == "imagenet" else 10


def _images(case, seed, batch):
    x = _randn(seed, 1, batch, 3, case["res"], case["res"]).to(torch.bfloat16)
    return x.contiguous(memory_format=torch.channels_last)


def _labels(seed, batch, classes):
    return torch.randint(0, classes, (batch,), device="cuda", generator=_generator(seed, 2))


def _resnet(case, seed):
    torch.manual_seed(seed)
    make = imagenet_resnet if case["dataset"] == "imagenet" else cifar_resnet
    return make(case["size"], 1, _classes(case))


def _norms(model):
    return [m for m in model.modules() if isinstance(m, torch.nn.BatchNorm2d)]


def prepare(case, seed):
    return {"train": _prepare_train, "sequence": _prepare_sequence, "evaluate": _prepare_evaluate,
            "allreduce": _prepare_allreduce, "dense": _prepare_dense}[case["kind"]](case, seed)


def _train_state(step, x, y, updated):
    """The step's inputs and the buffers, beside the loss, that it leaves its results in."""
    return {"kind": "train", "step": step, "x": x, "y": y, "updated": [b.w32 for b in step.opt.buckets] + updated}


def _prepare_train(case, seed):
    group = es.init()
    lars = (lambda ps, **kw: LARS(ps, lr=kw["lr"], momentum=0.9, weight_decay=1e-4)) if case["optimizer"] == "lars" else None
    step = TrainStep(_resnet(case, seed), group, mode=case["mode"], lr=0.1, momentum=0.9, weight_decay=1e-4,
                     inner_optimizer=lars)
    x, y = _images(case, seed, case["batch"]), _labels(seed, case["batch"], _classes(case))
    # the running statistics of all layers as views of one tensor, so that they can be handed out together
    norms = _norms(step.model)
    running = torch.empty(2, sum(m.num_features for m in norms), device="cuda")
    at = 0
    for m in norms:
        for row, name in ((0, "running_mean"), (1, "running_var")):
            view = running[row, at:at + m.num_features]
            view.copy_(getattr(m, name))
            setattr(m, name, view)
        at += m.num_features
    if case["graph"]:
        step.capture(x, y)
    # The fp32 master weights carry every gradient of the step (at the recipes' learning rate).  The momentum buffers are
    # left out: in a random-init ResNet a single bf16 rounding that falls the other way (sums meet in atomics) moves
    # the early layers' gradients by several per cent, from one run of the same code to the next.
    return _train_state(step, x, y, [running])


def _prepare_sequence(case, seed):
    group = es.init()
    torch.manual_seed(seed)
    step = TrainStep(LSTMClassifier(FRAME_FEATURES, case["hidden"], 2, VIDEO_CLASSES), group, mode="majority", lr=0.01,
                     momentum=0.9, weight_decay=1e-4)
    x = _randn(seed, 1, case["batch"], case["frames"], FRAME_FEATURES).to(torch.bfloat16)
    return _train_state(step, x, _labels(seed, case["batch"], VIDEO_CLASSES), [b.mom for b in step.opt.buckets])


def _prepare_evaluate(case, seed):
    model = prepare_model(_resnet(case, seed), torch.device("cuda", torch.cuda.current_device()))
    # a trained network's normalisation: no scale is zero, and the running statistics fit the activations
    for i, m in enumerate(_norms(model)):
        if not bool(m.weight.any()):
            m.weight.data.copy_(0.2 + 0.2 * torch.rand(m.num_features, device="cuda", generator=_generator(seed, 100 + i)))
        m.momentum = 1.0
    with torch.no_grad():
        model.train()
        model(_images(case, seed + 500000, 16))
    for m in _norms(model):
        m.momentum = 0.003
    model.eval()
    return {"kind": "evaluate", "model": model, "x": _images(case, seed, case["batch"])}


def _prepare_allreduce(case, seed):
    group = es.init()
    dtype = getattr(torch, case["dtype"])
    grad = (_randn(seed, 1, case["count"]) * 1e-2).to(dtype)
    out = torch.empty_like(grad)
    ar = es.PartialAllreduce(grad, group, mode=case["mode"], limiter=32, out=out).start()
    return {"kind": "allreduce", "ar": ar, "out": out}


def _prepare_dense(case, seed):
    m, n, k = case["rows"], case["outputs"], case["inputs"]
    x = _randn(seed, 1, m, k).to(torch.bfloat16).requires_grad_()
    w = (_randn(seed, 2, n, k) / math.sqrt(k)).to(torch.bfloat16).requires_grad_()
    b = (_randn(seed, 3, n) * 0.1).to(torch.bfloat16).requires_grad_() if case["bias"] else None
    return {"kind": "dense", "x": x, "w": w, "b": b, "dy": _randn(seed, 4, m, n) / m}


# ---------------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "train":
        return [state["step"].run_device(state["x"], state["y"])] + state["updated"]
    if kind == "evaluate":
        with torch.no_grad():
            return state["model"](state["x"])
    if kind == "allreduce":
        ar = state["ar"]
        ar.post()
        info = ar.wait()
        return {"out": state["out"], "contributors": info["contributors"], "applied": info["applied"]}
    y = ops.linear(state["x"], state["w"], state["b"])
    leaves = [t for t in (state["x"], state["w"], state["b"]) if t is not None]
    return [y.detach()] + list(torch.autograd.grad(y, leaves, state["dy"]))


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _convolutions(dataset, size, res):
    """(output pixels, multiply-adds per output pixel, is the stem) of every convolution and of the dense layer, per image,
    and the number of parameters."""
    if dataset == "imagenet":
        kind, blocks = IMAGENET_BLOCKS[size]
        width, first, strides = 64, (7, 2), [1, 2, 2, 2]
    else:
        kind, blocks = "building", [(size - 2) // 6] * 3
        width, first, strides = 16, (3, 1), [1, 2, 2]
    side = (res + first[1] - 1) // first[1]
    layers = [(side * side, 3 * first[0] ** 2 * width, True)]
    params = 3 * first[0] ** 2 * width + 2 * width
    if dataset == "imagenet":
        side = (side + 1) // 2
    cin = width
    for i, n in enumerate(blocks):
        f = width << i
        for j in range(n):
            s = strides[i] if j == 0 else 1
            out = (side + s - 1) // s
            cout = 4 * f if kind == "bottleneck" else f
            if kind == "bottleneck":
                convs = [(side, cin * f, f), (out, 9 * f * f, f), (out, f * cout, cout)]
            else:
                convs = [(out, 9 * cin * f, f), (out, 9 * f * f, f)]
            if j == 0:
                convs.append((out, cin * cout, cout))
            for d, macs, ch in convs:
                layers.append((d * d, macs, False))
                params += macs + 2 * ch
            side, cin = out, cout
    classes = 1000 if dataset == "imagenet" else 10
    layers.append((1, cin * classes, False))
    return layers, params + cin * classes + classes


def work(case):
    kind = case["kind"]
    if kind in ("train", "evaluate"):
        layers, params = _convolutions(case["dataset"], case["size"], case["res"])
        forward = 2.0 * case["batch"] * sum(p * m for p, m, _ in layers)
        stem = 2.0 * case["batch"] * sum(p * m for p, m, s in layers if s)
        images = 2.0 * case["batch"] * 3 * case["res"] ** 2
        if kind == "evaluate":
            return {"bytes": images + 2.0 * params + 4.0 * case["batch"] * _classes(case), "flops": forward}
        # master weights and momentum are read and written, the working copy is read and written
        return {"bytes": images + params * (4 + 4 + 4 + 4 + 2 + 2.0), "flops": 3 * forward - stem}
    if kind == "sequence":
        t, b, h, f = case["frames"], case["batch"], case["hidden"], FRAME_FEATURES
        rows, gates = t * b, 4 * h
        flops = 2.0 * rows * gates * (2 * (f + h) + 3 * 2 * h + h)   # the first layer's input takes no gradient
        params = gates * (f + h) + gates * 2 * h + 2 * gates + h * VIDEO_CLASSES + VIDEO_CLASSES
        return {"bytes": 2.0 * rows * f + params * (4 + 4 + 4 + 4 + 2 + 2.0), "flops": flops}
    if kind == "allreduce":
        return {"bytes": 2.0 * case["count"] * (4 if case["dtype"] == "float32" else 2), "flops": float(case["count"])}
    m, n, k = case["rows"], case["outputs"], case["inputs"]
    return {"bytes": 2.0 * 2 * (m * k + n * k) + 2 * 4.0 * m * n, "flops": 3 * 2.0 * m * n * k}


def tolerance(case):
    if case["kind"] == "allreduce":
        return "exact"           # one contributor: its own gradient, to the bit
    if case["kind"] == "dense":
        return {"rel": 5e-3}     # bf16 gradients, one rounding each; the fp32 output agrees far better
    if case["kind"] == "sequence":
        return {"rel": 1e-2}     # momentum buffers, that is gradients through bf16 gates and states
    if case["kind"] == "train":
        # loss, updated fp32 weights and running statistics of a network that computes in bf16: a few per cent of an update
        # that is a thousandth of the weights, and the loss of a small batch
        return {"rel": 1e-3}
    return {"rel": 2e-2}         # logits at the end of up to 53 layers of bf16 activations
