"""Workloads of this library for timing and comparing builds: the calls a training program makes, over the range of sizes it
makes them with.  One GPU, one worker (the fused reducers then run their single-worker path).

Four kinds of case:

``step``    one training step through ``GraphedStep``: forward, loss and metrics, backward, compressed reduce, SGD.  This is what
            ``bench.py`` and the trainer run; models and batch sizes are those of the zoo's two headline families.
``eval``    the forward pass of an evaluation batch (``CIFAR.test`` runs one per 256 test images; the last batch is ragged).
``reduce``  one ``Reducer.reduce`` call, with the gradient held in one of the three ways programs hold it:
            "arena"    parameter gradients of a model as views of a ``FlatArena``, reduced in place (the trainer's call);
            "tensors"  separately allocated send buffers and gradients of a model (the reference's calling convention);
            "single"   one tensor of n elements (the micro-benchmark's 1 K .. 64 M).
``codec``   ``compress`` and ``decompress`` of a compressor on one tensor, used without a reducer.
"""
from __future__ import annotations

import math

import torch

from gradient_compression_b200 import compressors, make_reducer, models, ops
from gradient_compression_b200.parallel import FlatArena, FlatSGD
from gradient_compression_b200.parallel.graph import GraphedStep
from gradient_compression_b200.train import CIFAR

DEVICE = "cuda"

# The reducers of the headline comparison, with the settings they are quoted with.
METHODS = {
    "allreduce": ("NoneAllReducer", {}),
    "qsgd-mn-2": ("QSGDMaxNormReducer", {"quantization_level": 2}),
    "qsgd-mn-4": ("QSGDMaxNormReducer", {"quantization_level": 4}),
    "qsgd-mn-8": ("QSGDMaxNormReducer", {"quantization_level": 8}),
    "qsgd-mn-ts-2-6": ("QSGDMaxNormTwoScaleReducer", {"quantization_level": 2, "higher_quantization_level": 6}),
    "qsgd-mn-ts-6-10": ("QSGDMaxNormTwoScaleReducer", {"quantization_level": 6, "higher_quantization_level": 10}),
    "grandk-mn-8": ("GlobalRandKMaxNormReducer", {"K": 10000, "quantization_level": 8}),
    "grandk-mn-ts-2-6": ("GlobalRandKMaxNormTwoScaleReducer", {"K": 10000, "quantization_level": 2, "higher_quantization_level": 6}),
    "topk-1pct": ("TopKReducerRatio", {"compression": 0.01}),
    "global-topk": ("GlobalTopKReducer", {"K": 10000}),
    "powersgd-1": ("RankKReducer", {"rank": 1}),
    "powersgd-2": ("RankKReducer", {"rank": 2}),
    "powersgd-4": ("RankKReducer", {"rank": 4}),
}
STEP_METHODS = ("allreduce", "qsgd-mn-8", "qsgd-mn-ts-6-10", "grandk-mn-8")
# The gradient of a network at its random initialisation is badly conditioned (a ReLU whose input is rounded to the other side of
# zero switches a whole path off: TF32 products summed in another order move it by several percent), and a captured step draws
# its rounding noise from the number of launches the process has made.  Steps are therefore compared by the loss, the running
# statistics and the parameters that the gradient updates, at a learning rate as near the end of the cosine schedule.
LEARNING_RATE = 1e-3
CODECS = ("QSGDMaxNormCompressor", "QSGDMaxNormTwoScaleCompressor", "QSGDWECModCompressor", "TernGradModCompressor")


def listed():
    return [
        # the headline of bench.py: ResNet-50, QSGD-MaxNorm 8 bit, batch 128
        {"name": "step-resnet50-qsgd8-b128", "kind": "step", "model": "ResNet50", "method": "qsgd-mn-8", "batch": 128},
        # the second headline model, in the communication-bound configuration, uncompressed
        {"name": "step-vgg16-allreduce-b128", "kind": "step", "model": "VGG16", "method": "allreduce", "batch": 128},
        # a small per-GPU batch, as when the global batch is spread over many workers: many short kernels
        {"name": "step-resnet18-allreduce-b31", "kind": "step", "model": "ResNet18", "method": "allreduce", "batch": 31},
        # the test pass after every epoch, at its default batch size
        {"name": "eval-resnet50-b256", "kind": "eval", "model": "ResNet50", "batch": 256},
        # the trainer's eager reduce of a whole model
        {"name": "reduce-arena-resnet50-qsgd8", "kind": "reduce", "layout": "arena", "model": "ResNet50", "method": "qsgd-mn-8"},
        # the reference's calling convention: send buffers and gradients allocated one by one
        {"name": "reduce-tensors-vgg16-ts", "kind": "reduce", "layout": "tensors", "model": "VGG16", "method": "qsgd-mn-ts-6-10"},
        {"name": "reduce-tensors-vgg16-powersgd2", "kind": "reduce", "layout": "tensors", "model": "VGG16", "method": "powersgd-2"},
        # layer-wise sparsification with error feedback: 161 tensors from 64 to 2.4 M elements
        {"name": "reduce-arena-resnet50-topk", "kind": "reduce", "layout": "arena", "model": "ResNet50", "method": "topk-1pct"},
        # the smallest call of the micro-benchmark: launches and host time only
        {"name": "reduce-single-1k-qsgd4", "kind": "reduce", "layout": "single", "n": 1024, "method": "qsgd-mn-4"},
        # shared random coordinates of an odd-sized vector
        {"name": "reduce-single-4m-grandk", "kind": "reduce", "layout": "single", "n": 4000037, "method": "grandk-mn-8"},
        # the largest call of the micro-benchmark
        {"name": "reduce-single-64m-qsgd8", "kind": "reduce", "layout": "single", "n": 1 << 26, "method": "qsgd-mn-8"},
        # encode and decode without a reducer
        {"name": "codec-qsgd4-1m", "kind": "codec", "codec": "QSGDMaxNormCompressor", "bits": 4, "n": 1048573},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("step", "eval", "reduce", "codec"), weights=(3, 1, 6, 2))[0]
    if kind == "step":
        model = rng.choice(("ResNet18", "ResNet34", "ResNet50", "VGG11", "VGG13", "VGG16", "VGG19"))
        return {"kind": kind, "model": model, "method": rng.choice(STEP_METHODS), "batch": _log_size(rng, 24, 128)}
    if kind == "eval":
        return {"kind": kind, "model": rng.choice(("ResNet18", "ResNet50", "VGG16")), "batch": _log_size(rng, 16, 256)}
    if kind == "codec":
        codec = rng.choice(CODECS)
        return {"kind": kind, "codec": codec, "bits": 1 if "Tern" in codec else rng.choice((2, 4, 6, 8)), "n": _log_size(rng, 1 << 10, 1 << 25)}
    layout = rng.choice(("arena", "tensors", "single", "single"))
    method = rng.choice([m for m in METHODS if m != "allreduce" or layout == "tensors"])
    if layout == "single":
        return {"kind": kind, "layout": layout, "n": _log_size(rng, 1 << 10, 1 << 26), "method": method}
    names = ("ResNet18", "ResNet50", "VGG16", "VGG19") if layout == "arena" else ("ResNet18", "VGG11", "VGG13", "VGG16")
    return {"kind": kind, "layout": layout, "model": rng.choice(names), "method": method}


# ------------------------------------------------------------------------------------------------ what a case works on
def _meta_model(name):
    with torch.device("meta"):
        return getattr(models, name)()


def _shapes(case):
    if case["layout"] == "single":
        if case["method"].startswith("powersgd"):         # a square matrix view of the vector, as the micro-benchmark has it
            side = math.isqrt(case["n"])
            return [(side, side)]
        return [(case["n"],)]
    return [tuple(p.shape) for p in _meta_model(case["model"]).parameters()]


_forward_flops = {}


def _flops(model):
    """Multiply-adds of one image's forward pass, times two."""
    if model not in _forward_flops:
        total = [0]

        def conv(m, _, out):
            total[0] += 2 * out.numel() * m.weight[0].numel()

        net = _meta_model(model).eval()
        for m in net.modules():
            if isinstance(m, (torch.nn.Conv2d, torch.nn.Linear)):
                m.register_forward_hook(conv)
        with torch.no_grad():
            net(torch.empty(1, 3, 32, 32, device="meta"))
        _forward_flops[model] = total[0]
    return _forward_flops[model]


def _n_params(model):
    return sum(p.numel() for p in _meta_model(model).parameters())


def _gradients(shapes, gen):
    """Gradient-like values: normal within a tensor, tensors of a model differing in scale by up to a factor of a hundred."""
    scales = [1e-3] if len(shapes) == 1 else [10.0 ** e for e in (torch.rand(len(shapes), generator=gen, device=DEVICE) * 2 - 4).tolist()]
    return [torch.randn(s, generator=gen, device=DEVICE) * k for s, k in zip(shapes, scales)]


# ------------------------------------------------------------------------------------------------ preparation
def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    return {"step": _prepare_step, "eval": _prepare_eval, "reduce": _prepare_reduce, "codec": _prepare_codec}[case["kind"]](case, seed, gen)


def _task(case, seed, gen):
    task = CIFAR(DEVICE, None, case["model"], seed=seed, data="synthetic", synthetic_train_size=1, synthetic_test_size=1)
    x = torch.randn(case["batch"], 3, 32, 32, device=DEVICE, generator=gen).contiguous(memory_format=torch.channels_last)
    return task, (x, torch.randint(0, 10, (case["batch"],), device=DEVICE, generator=gen))


def _prepare_step(case, seed, gen):
    task, batch = _task(case, seed, gen)
    name, config = METHODS[case["method"]]
    opt = FlatSGD(task.arena, lr=0.0, momentum=0.9, weight_decay=5e-4, nesterov=True)
    step = GraphedStep(task, make_reducer(name, DEVICE, None, dict(config, seed=seed)), opt)
    for _ in range(5):                       # eager steps, then the capture; at a learning rate of zero the parameters stay put
        step(batch)
    # other reducers of this process take their rounding noise from their own step counters, not from the launch counter
    step._set_step_from_device(False)
    opt.set_lr(LEARNING_RATE)
    task.arena.flat_momentum.zero_()
    running = [(n, b) for n, b in task.model.named_buffers() if n.endswith(("running_mean", "running_var"))]
    if len(running) > 60:
        running = [(n, b) for n, b in running if n.endswith("running_var")]
    return {"run": _run_step, "step": step, "batch": batch, "out": {"params": task.arena.flat_params, "running": [b for _, b in running]}}


def _prepare_eval(case, seed, gen):
    task, batch = _task(case, seed, gen)
    norms = [m for m in task.model.modules() if isinstance(m, torch.nn.BatchNorm2d)]
    for m in norms:
        m.momentum = 1.0                     # running statistics as training leaves them: those of the data
    task.batch_loss(batch)
    for m in norms:
        m.momentum = 0.1
    task.model.eval()
    return {"run": _run_eval, "task": task, "batch": batch}


def _prepare_reduce(case, seed, gen):
    name, config = METHODS[case["method"]]
    reducer = make_reducer(name, DEVICE, None, dict(config, seed=seed))
    if case["layout"] == "arena":
        net = getattr(models, case["model"])().to(DEVICE).to(memory_format=torch.channels_last)
        arena = FlatArena(net.parameters())
        send = out = arena.grads()
        for dst, src in zip(send, _gradients([t.shape for t in send], gen)):
            dst.copy_(src)
        result = [arena.flat_grads]
    else:
        arena = None
        send = _gradients(_shapes(case), gen)
        result = out = [torch.zeros_like(t) for t in send]
    return {"run": _run_reduce, "reducer": reducer, "send": send, "out": out, "result": result, "arena": arena}


def _prepare_codec(case, seed, gen):
    cls, noise = getattr(compressors, case["codec"]), compressors.NoiseSource(seed)
    if case["codec"].startswith("Tern"):
        codec = cls(DEVICE, noise=noise)
    elif "TwoScale" in case["codec"]:
        codec = cls(DEVICE, case["bits"], case["bits"] + 4, noise=noise)
    else:
        codec = cls(DEVICE, case["bits"], noise=noise)
    run = _run_two_scale if "TwoScale" in case["codec"] else _run_max_norm if "MaxNorm" in case["codec"] else _run_own_norm
    return {"run": run, "codec": codec, "x": torch.randn(case["n"], device=DEVICE, generator=gen) * 1e-3}


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    return state["run"](state)


def _run_step(s):
    loss = s["step"](s["batch"])
    return dict(s["out"], loss=loss)


def _run_eval(s):
    with torch.no_grad():
        x, y = s["batch"]
        logits = s["task"].model(x)
        metrics = s["task"].evaluate_predictions(logits, y)
    return {"logits": logits, "loss": metrics["cross_entropy_loss"]}


def _run_reduce(s):
    bits = s["reducer"].reduce(s["send"], s["out"])
    out = {"bits": bits, "grads": s["result"]}
    if (memory := getattr(s["reducer"], "_memory", None)) is not None:          # error feedback carried to the next step
        out["memory"] = memory
    return out


def _run_max_norm(s):
    norm = ops.absmax(s["x"])
    levels = s["codec"].compress(norm, s["x"])
    return {"norm": norm, "levels": levels, "values": s["codec"].decompress(norm, levels)}


def _run_two_scale(s):
    codec = s["codec"]
    norm = ops.absmax(s["x"])
    codec.begin()
    lower = codec.compress_lower(norm, s["x"])
    higher, mask = codec.compress_higher(norm, s["x"])
    levels = torch.where(mask.bool(), higher, lower)
    return {"norm": norm, "levels": levels, "mask": mask, "values": codec.decompress(norm, levels, mask)}


def _run_own_norm(s):
    norm, levels = s["codec"].compress(s["x"])
    return {"norm": norm, "levels": levels, "values": s["codec"].decompress(norm, levels)}


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Each input read once, each output and each piece of updated state written once; multiply-adds counted as two."""
    if case["kind"] == "step":                # parameters and momentum in and out, the gradient out, the batch in
        return {"bytes": 20 * _n_params(case["model"]) + 12296 * case["batch"], "flops": 3 * _flops(case["model"]) * case["batch"]}
    if case["kind"] == "eval":
        return {"bytes": 4 * _n_params(case["model"]) + 12336 * case["batch"], "flops": _flops(case["model"]) * case["batch"]}
    if case["kind"] == "codec":
        level = 1 if case["bits"] < 8 else 4
        return {"bytes": case["n"] * (8 + level + ("TwoScale" in case["codec"])), "flops": 0}
    shapes, method = _shapes(case), case["method"]
    n = sum(math.prod(s) for s in shapes)
    if method.startswith("powersgd"):
        rank = int(method[-1])
        matrices = [(s[0], math.prod(s[1:])) for s in shapes if len(s) > 1]
        return {"bytes": 16 * n, "flops": sum(6 * a * b * min(a, b, rank) for a, b in matrices)}
    if "topk" in method:                      # gradient and error memory in, both out
        return {"bytes": 16 * n, "flops": 0}
    if method.startswith("grandk") and case["layout"] == "arena":       # in place: only the selected coordinates move
        return {"bytes": 8 * min(n, 10000), "flops": 0}
    return {"bytes": 8 * n, "flops": 0}


def tolerance(case):
    if case["kind"] in ("step", "eval"):      # convolutions multiply in TF32 (10-bit mantissa), tens of layers deep
        return {"rel": 1e-2, "max": 0.5}
    if case["kind"] == "reduce" and case["method"].startswith("powersgd"):      # fp32 sums of up to 8192 products
        return {"rel": 3e-5, "max": 2e-3}
    return "exact"                            # seeded rounding noise and exact selection: the same bits everywhere
