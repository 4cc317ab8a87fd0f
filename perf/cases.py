"""The calls whose speed this library is judged by: hinge forests as programs use them.

Every case is a module of `RandomHingeForest` with the constructor's own random initialisation, called under
`torch.no_grad()` (op "predict") or called and differentiated through autograd (the other ops, one training step without
the optimizer).  Fields of a case:

  op      "predict", "train": a forest or fern;  "linear": forest with its fused linear layer;  "conv": convolutional trees;
          "pipeline": Linear -> BatchNorm1d -> forest with sequential ordinals
  kind    "tree" or "fern"
  B C K   samples, channels and inner positions per sample (K = 1: tabular data, x is [B, C]; else x is [B, C, H, W])
  T depth trees and their depth;  M: `extra_outputs` (0: none, a leaf holds one number)
  grad_x  whether the data take a gradient (a forest behind other layers) or not (a forest on the data set itself)
  dtype   "f32" or "f64";  deterministic: torch.use_deterministic_algorithms
"""
import math

import torch

from hingetreefortorch_b200 import RandomHingeForest as R

DEVICE = "cuda"


def _case(name, op, **fields):
    case = {"name": name, "op": op, "kind": "tree", "B": 1, "C": 1, "K": 1, "T": 1, "depth": 1, "M": 0, "grad_x": op != "predict",
            "dtype": "f32", "deterministic": False, "data": "normal"}
    case.update(fields)
    return case


def listed():
    return [
        # one request of a service: a small batch through a trained forest
        _case("predict_small", "predict", B=100, C=1000, T=100, depth=7, data="uniform"),
        # the operator's speed test: the smallest training step, launches and host work count
        _case("train_small", "train", B=100, C=1000, T=100, depth=7, M=1, data="uniform"),
        # an ordinary training step of ferns with several outputs per leaf
        _case("train_ferns", "train", kind="fern", B=4096, C=256, T=500, depth=10, M=10),
        # an ordinary training step at sizes that divide by nothing
        _case("train_odd_sizes", "train", B=10007, C=333, T=257, depth=9, M=3),
        # scoring of a large data set
        _case("predict_large", "predict", B=1048576, C=128, T=1024, depth=8),
        # full-batch training on the same data
        _case("train_large", "train", B=1048576, C=128, T=1024, depth=8),
        # image segmentation: a forest behind convolutions, 8 x 8 outputs per leaf at every position
        _case("train_images", "train", B=8, C=100, K=1024, T=100, depth=7, M=64),
        # reproducible training on the data set itself, one output per class
        _case("train_deterministic", "train", B=8192, C=784, T=100, depth=7, M=10, grad_x=False, deterministic=True, data="uniform"),
        # double precision, for small scientific data sets and gradient checks
        _case("train_double", "train", B=4096, C=64, T=200, depth=6, M=1, dtype="f64"),
        # forest with the class scores formed by its own linear layer
        _case("train_fused_linear", "linear", B=262144, C=784, T=100, depth=7, O=10),
        # a convolutional layer of trees, 3 x 3
        _case("train_conv2d", "conv", B=64, C=64, H=64, dims=2, window=3, stride=1, padding=1, T=128, depth=5),
        # sequential initialisation: learned projection to one feature per decision, normalised, then the forest
        _case("train_pipeline", "pipeline", B=8192, C=784, T=100, depth=7, grad_x=False, data="uniform"),
    ]


# ---- further cases of the same ranges ------------------------------------------------------------------------------

def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _down(value, limit, per_unit):
    """`value`, or what keeps value * per_unit within the limit."""
    return max(1, min(value, int(limit // max(1, per_unit))))


def draw(rng):
    op = rng.choice(["predict"] * 5 + ["train"] * 8 + ["linear"] * 2 + ["conv"] * 3 + ["pipeline"] * 2)
    kind = "fern" if rng.random() < 0.25 else "tree"
    if op in ("predict", "train"):
        depth = rng.randint(3, 10)
        M = rng.choice([0, 0, 0, 1, 2, 3, 5, 8, 10, 16, 26, 64])
        T = _down(_log(rng, 8, 1024), 1 << 23, (1 << depth) * max(1, M))
        C = _log(rng, 16, 2048)
        K = rng.choice([1, 1, 1, rng.randint(8, 64) ** 2])
        case = _case("", op, kind=kind, T=T, depth=depth, M=M, C=C, K=K, grad_x=op == "train" and rng.random() < 0.7)
        evals, rows = 1 << 28, 1 << 20
        if op == "train" and rng.random() < 0.2:  # ordered sums and wide numbers are used on small data sets
            case["dtype" if rng.random() < 0.5 else "deterministic"] = "f64" if rng.random() < 0.5 else True
            case["dtype"] = "f64" if case["dtype"] != "f32" else "f32"
            case["deterministic"] = case["dtype"] == "f32"
            evals, rows = 1 << 22, 16384
        B = _log(rng, 32, rows)
        B = _down(B, rows, K)
        B = _down(B, 1 << 27, C * K)
        B = _down(B, evals, T * K)
        case["B"] = _down(B, 1 << 29, T * K * max(1, M))
    elif op == "linear":
        depth, T, C, O = rng.randint(4, 8), _log(rng, 16, 256), _log(rng, 16, 1024), rng.randint(2, 16)
        B = _down(_log(rng, 64, 262144), 1 << 24, T)
        case = _case("", op, kind=kind, depth=depth, T=T, C=C, O=O, B=_down(B, 1 << 27, C), grad_x=rng.random() < 0.7)
    elif op == "conv":
        dims = rng.choice([1, 2, 2, 3])
        H = {1: _log(rng, 64, 4096), 2: _log(rng, 8, 96), 3: _log(rng, 6, 20)}[dims]
        window = rng.choice([2, 3, 3, 5]) if dims < 3 else rng.choice([2, 3])
        C, T = _log(rng, 1, 64), _log(rng, 4, 128)
        B = _down(_log(rng, 2, 64), 1 << (29 if dims < 3 else 26), C * T * H ** dims)
        case = _case("", op, kind=kind, dims=dims, H=H, window=window, stride=rng.choice([1, 1, 2]), padding=rng.choice([0, window // 2]),
                     depth=rng.randint(3, 7), C=C, T=T, B=B, M=rng.choice([0, 0, 0, 4]), grad_x=rng.random() < 0.8)
        if case["M"]:
            case["B"] = _down(B, 1 << 25, C * T * H ** dims)
    else:
        depth = rng.randint(4, 8)
        T = _log(rng, 16, 128)
        T += (-T) % 4  # the projection's width is a multiple of four
        if kind == "tree":
            T = _down(T, 16384, 1 << depth) // 4 * 4
        case = _case("", op, kind=kind, depth=depth, T=T, C=4 * _log(rng, 8, 256), B=_log(rng, 128, 16384), grad_x=rng.random() < 0.3)
    case["data"] = rng.choice(["normal", "uniform"])
    del case["name"]
    return case


# ---- inputs, the call, its results ---------------------------------------------------------------------------------

def _random(case, shape, generator, dtype):
    make = torch.rand if case["data"] == "uniform" else torch.randn
    return make(shape, generator=generator, device=DEVICE, dtype=dtype)


def _decisions(case):
    return case["depth"] if case["kind"] == "fern" else 2 ** case["depth"] - 1


def _module(case):
    fern, T, depth = case["kind"] == "fern", case["T"], case["depth"]
    extra = case["M"] if case["M"] > 0 else None
    if case["op"] == "conv":
        cls = getattr(R, "Hinge%sConv%dd" % ("Fern" if fern else "Tree", case["dims"]))
        return cls(case["C"], T, depth, case["window"], stride=case["stride"], padding=case["padding"], extra_outputs=max(1, case["M"]))
    if case["op"] == "linear":
        cls = R.RandomHingeFernFusedLinear if fern else R.RandomHingeForestFusedLinear
        return cls(case["C"], T, case["O"], depth)
    forest = R.RandomHingeFern if fern else R.RandomHingeForest
    if case["op"] == "pipeline":
        width = T * _decisions(case)
        return R.LinearBatchNormForest(R.LinearBatchNorm1d(case["C"], width), forest(width, T, depth, init_type="sequential"))
    if extra == 64:  # a patch of the segmentation, as the module takes it
        extra = [8, 8]
    return forest(case["C"], T, depth, extra_outputs=extra)


def _data_shape(case):
    if case["op"] == "conv":
        return [case["B"], case["C"]] + [case["H"]] * case["dims"]
    side = math.isqrt(case["K"])
    return [case["B"], case["C"]] + ([] if case["K"] == 1 else [side, case["K"] // side])


def prepare(case, seed):
    torch.manual_seed(seed)
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    module = _module(case).to(device=DEVICE, dtype=dtype)
    module.train(case["op"] != "predict")
    x = _random(case, _data_shape(case), generator, dtype)
    if case["op"] == "predict":
        return {"case": case, "module": module, "x": x}
    x.requires_grad_(case["grad_x"])
    wrt = ([x] if case["grad_x"] else []) + [p for p in module.parameters() if p.requires_grad]
    g = torch.randn(_out_shape(case), generator=generator, device=DEVICE, dtype=dtype)
    return {"case": case, "module": module, "x": x, "wrt": wrt, "g": g}


def _out_positions(case):
    """Output positions per sample of a convolution."""
    return ((case["H"] + 2 * case["padding"] - case["window"]) // case["stride"] + 1) ** case["dims"]


def _out_shape(case):
    if case["op"] == "linear":
        return [case["B"], case["O"]]
    if case["op"] == "conv":
        side = (case["H"] + 2 * case["padding"] - case["window"]) // case["stride"] + 1
        return [case["B"], case["T"]] + [side] * case["dims"] + ([case["M"]] if case["M"] > 1 else [])
    shape = [case["B"], case["T"]] + _data_shape(case)[2:]
    return shape + ([8, 8] if case["M"] == 64 else [case["M"]] if case["M"] > 0 else [])


def _step(state):
    out = state["module"](state["x"])
    results = [out.detach()] + list(torch.autograd.grad(out, state["wrt"], state["g"]))
    if state["case"]["op"] == "pipeline":
        front = state["module"].front
        results += [front.running_mean, front.running_var]
    return results


def run(state):
    case = state["case"]
    if case["op"] == "predict":
        with torch.no_grad():
            return state["module"](state["x"])
    if not case["deterministic"]:
        return _step(state)
    torch.use_deterministic_algorithms(True)
    try:
        return _step(state)
    finally:
        torch.use_deterministic_algorithms(False)


def work(case):
    """Bytes: data, parameters and upstream gradient read once, result and gradients written once.  Operations: a subtraction and
    a comparison per decision, a product per output, three per output in the backward, and the products of dense layers."""
    size = 8 if case["dtype"] == "f64" else 4
    B, T, N, M = case["B"], case["T"], _decisions(case), max(1, case["M"])
    x = math.prod(_data_shape(case))
    out = math.prod(_out_shape(case))
    trees = T * case["C"] if case["op"] == "conv" else T
    thresholds, weights = trees * N, trees * 2 ** case["depth"] * M
    evals = B * (trees * _out_positions(case) if case["op"] == "conv" else T * case["K"])
    bytes_ = size * (x + thresholds + weights + out) + 8 * thresholds
    flops = evals * (2 * case["depth"] + M)
    if case["op"] != "predict":
        bytes_ += size * (out + thresholds + weights + (x if case["grad_x"] else 0))
        flops += 3 * evals * M
    if case["op"] == "linear":
        bytes_ += 2 * size * (T + 1) * case["O"]
        flops += 6 * B * T * case["O"]
    if case["op"] == "pipeline":  # the activations between the two layers need not leave the chip for the count
        width = T * N
        bytes_ += 2 * size * case["C"] * width
        flops += (6 if case["grad_x"] else 4) * B * case["C"] * width
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # A prediction is one product per value; the fixed-order mode fixes every sum.
    if case["op"] == "predict" or case["deterministic"]:
        return "exact"
    if case["dtype"] == "f64":
        return {"rel": 1e-12}
    # 19-bit products in the projection: another order of its sums sends a few samples through another branch, and each of
    # those moves a whole term of a gradient.
    if case["op"] == "pipeline":
        return {"rel": 1e-2, "max": 0.9}
    return {"rel": 1e-5}
