"""The work that users of this runtime have it do, through its public entry points.

Five families, each over the range its users meet:

  conv       one Convolution layer with bias and fused ReLU on device arrays (the single-layer configuration)
  resnet18   the ResNet-18 topology: fp32 on tensor cores, int8, and the CUDA-core fp32 mode that keeps the reference's
             own error budget; device arrays, pinned host arrays, or numpy arrays
  mobilenet  the MobileNetV2 topology (1x1 and depthwise layers, ReLU6)
  ip         one InnerProduct layer, fp32 and int8, from one row to 4096
  dynamic    a network with `?` extents, called with one image of any height and width through the shape-checked entry

Weights come from the repository's own model writers and stay the same; the seed makes the inputs, U(-1,1) as the
benchmark configurations state.  Every state owns its handle, as a program with one model in hand does.
"""
import importlib.util
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.getcwd()


def _package():
    """The package lives in a folder whose name is no Python identifier; the repository's entry file loads it."""
    spec = importlib.util.spec_from_file_location("repository_entry", os.path.join(ROOT, "__graft_entry__.py"))
    entry = importlib.util.module_from_spec(spec)
    sys.modules["repository_entry"] = entry
    spec.loader.exec_module(entry)
    return entry.load_package()


pkg = _package()
MODES = {"fp32": pkg.FP32_SPLIT, "int8": pkg.FP32_SPLIT, "exact": pkg.FP32_CUDA}
IMAGE = 224 * 224  # pixels of one image of the benchmark configurations


def listed():
    return [
        # the single-layer configuration as it stands: the smallest call, launches and their latency
        {"name": "conv_one", "family": "conv", "n": 1, "h": 56, "w": 56, "cin": 64, "cout": 64, "k": 3, "stride": 1},
        # the drop-in call: one image in, one result out, numpy arrays, as a compiled model's users call it
        {"name": "resnet18_one_host", "family": "resnet18", "n": 1, "size": 224, "data": "fp32", "entry": "host"},
        # the headline configuration, inputs resident on the GPU
        {"name": "resnet18_batch", "family": "resnet18", "n": 64, "size": 224, "data": "fp32", "entry": "device"},
        # the same end to end from pinned host memory, upload and download inside the call
        {"name": "resnet18_batch_pinned", "family": "resnet18", "n": 64, "size": 224, "data": "fp32", "entry": "pinned"},
        # results within the reference's own error budget: fp32 multiplies and sums on the CUDA cores
        {"name": "resnet18_exact", "family": "resnet18", "n": 8, "size": 224, "data": "exact", "entry": "device"},
        # the quantised network at its large batch
        {"name": "resnet18_int8", "family": "resnet18", "n": 256, "size": 224, "data": "int8", "entry": "device"},
        # a latency-bound service: one image, many small layers
        {"name": "mobilenet_one", "family": "mobilenet", "n": 1, "size": 224, "data": "fp32", "entry": "device"},
        # the batch that is sharded over the GPUs of a box
        {"name": "mobilenet_batch", "family": "mobilenet", "n": 256, "size": 224, "data": "fp32", "entry": "device"},
        # one row through a large layer: a pass over its weights
        {"name": "ip_row", "family": "ip", "m": 1, "k": 4096, "n": 4096, "data": "fp32"},
        # a quantised layer of odd extents
        {"name": "ip_ragged_int8", "family": "ip", "m": 200, "k": 1001, "n": 1537, "data": "int8"},
        # the largest layer of the sweep
        {"name": "ip_large", "family": "ip", "m": 4096, "k": 4096, "n": 4096, "data": "fp32"},
        # an image of whatever size it happens to have, through the entry with shapes and capacities
        {"name": "dynamic_odd", "family": "dynamic", "h": 211, "w": 173, "classes": 0},
    ]


def _log_int(rng, low, high):
    """A whole number spread evenly over the logarithm of [low, high]."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    family = rng.choice(["conv", "resnet18", "resnet18", "resnet18", "mobilenet", "mobilenet", "ip", "ip", "ip", "dynamic"])
    if family == "conv":
        # layers of ordinary networks: channels in eights, any image extent
        return {"family": "conv", "n": _log_int(rng, 1, 64), "h": _log_int(rng, 7, 112), "w": _log_int(rng, 7, 112),
                "cin": 8 * _log_int(rng, 2, 32), "cout": 8 * _log_int(rng, 2, 32), "k": rng.choice([1, 3]), "stride": rng.choice([1, 2])}
    if family in ("resnet18", "mobilenet"):
        data = rng.choice(["fp32", "fp32", "int8", "int8", "exact"]) if family == "resnet18" else "fp32"
        size = _log_int(rng, 64, 320)
        # never more pixels than the largest listed case of the kind
        most = (8 if data == "exact" else 256) * IMAGE / (size * size)
        return {"family": family, "n": _log_int(rng, 1, max(1, min(256, int(most)))), "size": size, "data": data,
                "entry": rng.choice(["device", "device", "pinned", "host"])}
    if family == "ip":
        m, k, n = _log_int(rng, 1, 4096), _log_int(rng, 512, 4096), _log_int(rng, 512, 4096)
        if rng.random() < 0.5:  # layer extents are whole sixteens as often as they are anything else
            k, n = k // 16 * 16, n // 16 * 16
        return {"family": "ip", "m": m, "k": k, "n": n, "data": rng.choice(["fp32", "int8"])}
    return {"family": "dynamic", "h": _log_int(rng, 32, 384), "w": _log_int(rng, 32, 384), "classes": rng.choice([0, 10])}


_FOLDER = None
_FILES = {}


def _files(case):
    """The model's .param and .bin, written once in a process: what a user has on disk."""
    global _FOLDER
    f = case["family"]
    # the batch, the entry and (but for int8 weights) the accuracy mode are no part of the model
    parts = {"conv": ("h", "w", "cin", "cout", "k", "stride"), "resnet18": ("size",), "mobilenet": ("size",), "ip": ("k", "n"), "dynamic": ("classes",)}
    int8 = case.get("data") == "int8"
    key = (f, int8) + tuple(case[p] for p in parts[f])
    if key not in _FILES:
        if _FOLDER is None:
            _FOLDER = tempfile.TemporaryDirectory(prefix="ncnn_b200_cases_")
        path = os.path.join(_FOLDER.name, "model%d" % len(_FILES))
        if f == "conv":
            _FILES[key] = pkg.zoo.single_conv(path, h=case["h"], w=case["w"], cin=case["cin"], cout=case["cout"], k=case["k"],
                                              stride=case["stride"], pad=case["k"] // 2)
        elif f == "resnet18":
            _FILES[key] = pkg.zoo.resnet18(path, int8=int8, size=case["size"])
        elif f == "mobilenet":
            _FILES[key] = pkg.zoo.mobilenet_v2(path, size=case["size"])
        elif f == "ip":
            _FILES[key] = pkg.zoo.inner_product(path, case["k"], case["n"], int8=int8)
        else:
            _FILES[key] = pkg.zoo.dynamic_convnet(path, classes=case["classes"])
    return _FILES[key]


def _uniform(shape, seed, device):
    g = torch.Generator(device=device).manual_seed(seed)
    return torch.rand(shape, generator=g, device=device) * 2 - 1


def prepare(case, seed):
    param, bin_ = _files(case)
    if case["family"] == "dynamic":
        x = _uniform((3, case["h"], case["w"]), seed, "cuda").cpu().numpy()
        return {"entry": "dynamic", "model": pkg.DynamicModel(param, bin_, [[3, None, None]]), "x": x}
    model = pkg.Model(param, bin_, accuracy_mode=MODES[case.get("data", "fp32")])
    count = case["m"] if case["family"] == "ip" else case["n"]
    entry = case.get("entry", "device")
    x = _uniform((count, *model.input_shapes[0]), seed, "cuda")
    state = {"entry": entry, "model": model, "count": count, "x": x}
    if entry == "host":
        state["x"] = x.cpu().numpy()
    elif entry == "pinned":
        state["x"] = x.cpu().pin_memory()
        state["y"] = torch.empty((count, *model.output_shapes[0])).pin_memory()
    else:
        state["y"] = torch.empty((count, *model.output_shapes[0]), device="cuda")
    return state


def run(state):
    entry, model = state["entry"], state["model"]
    if entry in ("host", "dynamic"):
        return model.run(state["x"])
    x, y = state["x"], state["y"]
    if entry == "pinned":
        status = model.run_raw(state["count"], [x.data_ptr()], [y.data_ptr()])
        if status != 0:
            raise RuntimeError("run_batch answered status %d" % status)
        return y
    model.run_device(state["count"], [x.data_ptr()], [y.data_ptr()], torch.cuda.current_stream().cuda_stream)
    return y


def _conv(h, w, k, stride, cin, cout, groups=1):
    """(multiply-adds, weights and biases, output height, output width) of a convolution padded by k // 2."""
    oh, ow = (h + 2 * (k // 2) - k) // stride + 1, (w + 2 * (k // 2) - k) // stride + 1
    weights = cout * (cin // groups) * k * k
    return oh * ow * weights, weights, cout, oh, ow


def _layers(case):
    """(multiply-adds of one item, weights, biases, input values, output values)."""
    macs = weights = biases = 0
    f = case["family"]

    def add(h, w, *conv, **more):
        nonlocal macs, weights, biases
        m, wt, b, oh, ow = _conv(h, w, *conv, **more)
        macs, weights, biases = macs + m, weights + wt, biases + b
        return oh, ow

    if f == "ip":
        return case["k"] * case["n"], case["k"] * case["n"], case["n"], case["k"], case["n"]
    if f == "conv":
        oh, ow = add(case["h"], case["w"], case["k"], case["stride"], case["cin"], case["cout"])
        return macs, weights, biases, case["cin"] * case["h"] * case["w"], case["cout"] * oh * ow
    if f == "dynamic":
        h, w = add(case["h"], case["w"], 3, 2, 3, 32)
        add(h, w, 3, 1, 32, 32)
        add(h, w, 3, 1, 32, 32)
        if case["classes"]:
            add(1, 1, 1, 1, 32, case["classes"])
            out = case["classes"]
        else:
            add(h, w, 1, 1, 32, 8)
            out = 8 * h * w
        return macs, weights, biases, 3 * case["h"] * case["w"], out
    size = case["size"]
    if f == "resnet18":
        h, w = add(size, size, 7, 2, 3, 64)
        h, w = (h - 1) // 2 + 1, (w - 1) // 2 + 1
        cin = 64
        for stage, c in enumerate((64, 128, 256, 512)):
            for block in range(2):
                stride = 2 if stage and not block else 1
                if stride == 2:
                    add(h, w, 1, 2, cin, c)
                h, w = add(h, w, 3, stride, cin, c)
                add(h, w, 3, 1, c, c)
                cin = c
        add(1, 1, 1, 1, 512, 1000)
    else:
        h, w = add(size, size, 3, 2, 3, 32)
        cin = 32
        for t, c, n, s in ((1, 16, 1, 1), (6, 24, 2, 2), (6, 32, 3, 2), (6, 64, 4, 2), (6, 96, 3, 1), (6, 160, 3, 2), (6, 320, 1, 1)):
            for i in range(n):
                hidden = cin * t
                if t != 1:
                    add(h, w, 1, 1, cin, hidden)
                h, w = add(h, w, 3, s if i == 0 else 1, hidden, hidden, groups=hidden)
                add(h, w, 1, 1, hidden, c)
                cin = c
        add(h, w, 1, 1, cin, 1280)
        add(1, 1, 1, 1, 1280, 1000)
    return macs, weights, biases, 3 * size * size, 1000


def work(case):
    """The caller's arrays once, the weights once in the precision of the model file, and every multiply-add."""
    macs, weights, biases, inputs, outputs = _layers(case)
    count = case["m"] if case["family"] == "ip" else case.get("n", 1)
    width = 1 if case.get("data") == "int8" else 4
    return {"bytes": 4.0 * count * (inputs + outputs) + width * weights + 4.0 * biases, "flops": 2.0 * macs * count}


def tolerance(case):
    """int8 sums are whole numbers and their rounding is fixed.  fp32 on tensor cores carries each operand as a pair of
    bf16 numbers (16 significant bits): 3e-6 to 1e-5 for a layer, 4e-5 to 6e-5 for a network of twenty to fifty layers."""
    data = case.get("data", "fp32")
    if data == "int8":
        return "exact"
    if data == "exact":
        return {"rel": 1e-5}
    return {"rel": 1e-4} if case["family"] in ("resnet18", "mobilenet") else {"rel": 3e-5}
