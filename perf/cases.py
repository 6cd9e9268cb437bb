"""Inference cases that stand for what users of this runtime have it do: a compiled model's call
sequence, replayed through ``occamy_b200.replay``.

``listed()`` names the cases that are looked at most, ``draw(rng)`` gives others of the same ranges.
A case says which graph runs (the benchmark graphs of ``occamy_b200.graphs``, or one convolution),
the batch and image size, the arithmetic mode, whether the call sequence was compiled with the
conv + bias + ReLU fusion, and where the batch comes from:

* ``io = "host"``: ``Program.run`` -- host batch in, host result out, complete on return.  This is a
  compiled model's own call sequence.
* ``io = "device"``: ``Program.run_raw`` with the batch already in HBM and the result left there, the
  call returning without a wait: a server that pipelines inferences.

The weights of a model are the same whatever the seed (a served model is loaded once and sees one
batch after another); the seed makes the images.
"""
from __future__ import annotations

from functools import lru_cache

import numpy as np
import torch

from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

MATH = {"fp32": rt.MATH_FP32, "bf16": rt.MATH_BF16, "fp16": rt.MATH_F16}


def _net(graph, batch, image, math, io, fuse, variant="v1"):
    return {"graph": graph, "variant": variant, "batch": batch, "image": image, "math": math,
            "io": io, "fuse": fuse}


def _conv(batch, channels, filters, size, window, stride, math, io):
    return {"graph": "single_conv", "batch": batch, "channels": channels, "filters": filters,
            "image": size, "window": window, "stride": stride, "math": math, "io": io, "fuse": 1}


def listed():
    return [
        # one fused Conv + bias + ReLU call, 64 -> 64 channels at 56 x 56: the smallest program a
        # compiler emits; latency and the host path count
        dict(_conv(1, 64, 64, 56, 3, 1, "bf16", "device"), name="conv_b1"),
        # batch 1, unfused, host in and host out: how the reference's own model scripts call it
        dict(_net("resnet50", 1, 224, "bf16", "host", 0), name="resnet50_b1_host_unfused"),
        # a server's small dynamic batch
        dict(_net("resnet50", 8, 224, "bf16", "device", 1), name="resnet50_b8"),
        # one GPU's share of batch 256 on eight GPUs
        dict(_net("resnet50", 32, 224, "bf16", "device", 1), name="resnet50_b32"),
        # a batch and an image size that nothing divides; stride on the 3x3 layers
        dict(_net("resnet50", 61, 201, "bf16", "device", 1, "v1.5"), name="resnet50_v15_b61_201px"),
        # the headline batch, resident
        dict(_net("resnet50", 256, 224, "bf16", "device", 1), name="resnet50_b256"),
        # the headline batch end to end: pinned host batch in, result back
        dict(_net("resnet50", 256, 224, "bf16", "host", 1), name="resnet50_b256_host"),
        # the mode for users who need the CPU's digits (1e-4)
        dict(_net("resnet50", 16, 224, "fp32", "device", 1), name="resnet50_b16_fp32"),
        # on-device style latency: one image through the small network
        dict(_net("mobilenet_v2", 1, 224, "fp16", "device", 1), name="mobilenet_v2_b1"),
        # the small network at its benchmark batch
        dict(_net("mobilenet_v2", 128, 224, "fp16", "device", 1), name="mobilenet_v2_b128"),
        # a few images through the network whose classifier holds most of the weights
        dict(_net("vgg16", 5, 224, "bf16", "device", 1), name="vgg16_b5"),
        # the same network at its benchmark batch
        dict(_net("vgg16", 64, 224, "bf16", "device", 1), name="vgg16_b64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["resnet50", "resnet50", "resnet50", "mobilenet_v2", "mobilenet_v2", "vgg16",
                       "fp32", "single_conv"])
    io = rng.choice(["device", "device", "host"])
    fuse = rng.choice([1, 1, 0])
    if kind == "single_conv":
        window = rng.choice([1, 3, 3])
        size = _log_int(rng, 7, 112)
        channels, filters = 8 * _log_int(rng, 2, 64), 8 * _log_int(rng, 2, 64)
        most = max(1, min(64, int(4e7 / (max(channels, filters) * size * size))))
        return _conv(_log_int(rng, 1, most), channels, filters, size, window, rng.choice([1, 1, 2]),
                     rng.choice(["bf16", "bf16", "fp16", "fp32"]), io)
    image = rng.randint(97, 256)
    scale = (224.0 / image) ** 2

    def batch(most):
        return _log_int(rng, 1, max(1, min(most, int(most * scale))))

    if kind == "fp32":
        return _net("resnet50", batch(16), image, "fp32", io, fuse, rng.choice(["v1", "v1.5"]))
    if kind == "resnet50":
        return _net("resnet50", batch(256), image, "bf16", io, fuse, rng.choice(["v1", "v1.5"]))
    if kind == "mobilenet_v2":
        return _net("mobilenet_v2", batch(128), image, "fp16", io, fuse)
    return _net("vgg16", batch(64), image, "bf16", io, fuse)


def _build(case, batch):
    if case["graph"] == "single_conv":
        r = case["window"]
        return graphs.single_conv(0, batch, case["channels"], case["image"], case["image"],
                                  case["filters"], r, r // 2, case["stride"])
    if case["graph"] == "resnet50":   # logits as the result: the softmax saturates on random weights
        return graphs.resnet50(batch, 0, case["variant"], softmax=False, image=case["image"])
    return getattr(graphs, case["graph"])(batch, 0, image=case["image"])


@lru_cache(maxsize=24)
def _graph(key):
    case = dict(key)
    return _build(case, case["batch"])


@lru_cache(maxsize=24)
def _program(key):
    """The compiled model: built once, called with one batch after another."""
    case = dict(key)
    program = _graph(key).to_program()
    program.lower(fuse=case["fuse"], dealloc_opt=True, pool_opt=True)
    return program


@lru_cache(maxsize=1)
def _binding():
    return replay.Binding()


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def prepare(case, seed):
    key = _key(case)
    g = _graph(key)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["graph"] == "single_conv":   # activations: U(-1, 1)
        x = torch.rand(g.input_shape, generator=gen, device="cuda") * 2.0 - 1.0
    else:                                # normalised images: N(0, 1)
        x = torch.randn(g.input_shape, generator=gen, device="cuda")
    rt.set_math_mode(MATH[case["math"]])
    state = {"program": _program(key), "binding": _binding(), "io": case["io"]}
    if case["io"] == "host":
        state["pinned"] = x.cpu().pin_memory()
        state["x"] = state["pinned"].numpy()
    else:
        state["x"] = x
        state["out"] = torch.empty(g.shapes[g.outputs[0]], device="cuda")
    torch.cuda.synchronize()
    return state


def run(state):
    if state["io"] == "host":
        return state["program"].run(state["binding"], state["x"])
    out = state["out"]
    state["program"].run_raw(state["binding"], state["x"].data_ptr(), 3, [out.data_ptr()], 3)
    return out


def work(case):
    """The images, the weights (two bytes each in the 16-bit modes) and the result, each moved once;
    multiply-adds of the convolutions and the classifier count as two operations."""
    g = _graph(_key(case))
    weights = sum(int(a.size) for a in g.consts.values())
    x, y = int(np.prod(g.input_shape)), int(np.prod(g.shapes[g.outputs[0]]))
    return {"bytes": 4 * x + (4 if case["math"] == "fp32" else 2) * weights + 4 * y,
            "flops": g.conv_flops()}


def tolerance(case):
    """One convolution: its result is rounded to the mode's 16-bit type once.  A network: every stored
    activation is rounded, and the roundings of some fifty layers add up."""
    if case["graph"] == "single_conv":
        return {"rel": {"bf16": 3e-3, "fp16": 5e-4, "fp32": 1e-5}[case["math"]]}
    return {"rel": {"bf16": 1e-2, "fp16": 1e-2, "fp32": 5e-5}[case["math"]]}
