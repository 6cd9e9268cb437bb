"""Large batches from host memory, which are computed in pieces while they arrive: every pass with another
batch, and with a constant that changes, against the same model computed from device memory."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from calls import Inference, rand
from helpers import max_rel_err
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt
from oracle import ref

pytestmark = pytest.mark.gpu

PASSES = 9


def net(N, size):
    g = graphs.Graph((N, 3, size, size), seed=N)
    v = g.relu(g.conv(0, *g.he_conv(64, 3, 7, 7), pads=(3, 3), strides=(2, 2)))
    v = g.maxpool(v, (3, 3), (1, 1), (2, 2))
    y = g.relu(g.conv(v, *g.he_conv(64, 64, 3, 3), pads=(1, 1)))
    v = g.relu(g.add(g.conv(y, *g.he_conv(64, 64, 1, 1)), v))
    g.mark_output(g.linear(g.flatten(g.gap(v)), 64, 40))
    return g


@pytest.mark.parametrize("fuse", [replay.FUSE_REFERENCE, replay.FUSE_NONE])
@pytest.mark.parametrize("math", [rt.MATH_BF16, rt.MATH_F16, rt.MATH_FP32])
@pytest.mark.parametrize("N,size", [(128, 112), (151, 121), (127, 112)])
def test_batches(binding, N, size, math, fuse):
    g = net(N, size)
    rt.set_math_mode(math)
    p = g.to_program()
    p.lower(fuse=fuse)
    rng = np.random.default_rng(N)
    xs = [rng.standard_normal(g.input_shape, dtype=np.float32) for _ in range(2)]
    head = max(g.consts, key=lambda k: g.consts[k].size == 64 * 40)
    for i in range(PASSES):
        if i == PASSES - 2:   # the classifier's weights, in place
            g.consts[head] *= 0.5
        x = torch.from_numpy(xs[i % 2] * (1 + i)).pin_memory()
        (got,) = p.run(binding, x.numpy())
        dev = x.cuda()
        want = torch.empty(g.shapes[g.outputs[0]], device="cuda")
        torch.cuda.synchronize()
        p.run_raw(binding, dev.data_ptr(), 3, [want.data_ptr()], 3)
        rt.synchronize()
        want = want.cpu().numpy()
        assert np.abs(got - want).max() <= {rt.MATH_FP32: 2e-5, rt.MATH_F16: 1e-3}.get(math, 8e-3) * np.abs(want).max()
    assert rt.last_error() == 0


def small_model(N, K=40):
    w, b, fc = rand(1, 16, 16, 3, 3, scale=0.1), rand(2, 16), rand(3, K, 16, scale=0.3)

    def run(x, between=None, mid=False):
        """x -> convolution, ReLU -> mean -> product; `between` the upload and the rest."""
        with Inference(8 * x.nbytes) as f:
            p = f.put(x)
            if between is not None:
                between()
            y, o = f.conv(p, x.shape, f.put(w), w.shape, f.put(b), (1, 1), act=1)
            m = f.place(N * 16 * 4)
            f.L.DNNReduceFunc(f.h, 4, y, rt.dims(o), m, rt.dims((N, 16, 1, 1)), 5)
            z, o = f.matmul(m, (N, 16), f.put(fc), fc.shape)
            return [f.get(z, o)] + ([f.get(m, (N, 16))] if mid else [])

    def want(x):
        m = ref.conv2d(x, w, b, (1, 1), act=1).mean((2, 3))
        return [m @ fc.T, m]
    return run, want


def test_wait_behind_the_upload(native_libs):
    """A wait right behind the upload is one for the upload: the host buffer may be used for something else then."""
    rt.set_math_mode(rt.MATH_BF16)
    N = 128
    run, want = small_model(N)
    xs = [rand(10 + i, N, 16, 96, 96) for i in range(2)]
    wants = [want(x)[0] for x in xs]
    buf = torch.empty(xs[0].shape).pin_memory().numpy()

    def refill():
        rt.synchronize()
        buf[-8:] = 0   # what is copied last
    for i in range(PASSES + 6):
        buf[...] = xs[i % 2]
        (got,) = run(buf, refill if i >= PASSES else None)
        assert max_rel_err(got, wants[i % 2]) <= 2e-2, i
    assert rt.last_error() == 0


def test_pieces_need_other_kernels(binding):
    """MobileNetV2 at batch 160: a piece of 40 images takes a block as one kernel that neither the whole batch nor the
    other pieces do.  Batches of other sizes share the packed weights in between."""
    rt.set_math_mode(rt.MATH_F16)
    rt.lib().occamy_clear_weight_cache()
    g = graphs.mobilenet_v2(batch=160, seed=1, image=224)
    programs = {}
    for n in (160, 40, 2):
        h = graphs.mobilenet_v2(batch=n, seed=1, image=224)
        assert list(h.consts) == list(g.consts)
        h.consts = g.consts   # the same host arrays
        programs[n] = h.to_program()
        programs[n].lower(fuse=replay.FUSE_REFERENCE)
    x = torch.from_numpy(rand(1, *g.input_shape)).pin_memory().numpy()
    first = {n: p.run(binding, x[:n])[0] for n, p in programs.items()}
    n0 = rt.form_counters()["in_pieces"]
    for i in range(10):
        for n in ((160, 2) if i < 6 else (160, 40, 2)):
            (got,) = programs[n].run(binding, x[:n])
            assert max_rel_err(got, first[n]) <= 5e-2, (i, n)
    assert rt.form_counters()["in_pieces"] > n0
    assert rt.last_error() == 0


@pytest.mark.parametrize("name,math,N,image", [("resnet50", rt.MATH_BF16, 160, 97), ("mobilenet_v2", rt.MATH_F16, 160, 128),
                                               ("vgg16", rt.MATH_BF16, 136, 112),
                                               # four pieces
                                               ("resnet50", rt.MATH_BF16, 208, 97), ("resnet50", rt.MATH_BF16, 253, 129),
                                               ("mobilenet_v2", rt.MATH_F16, 235, 112), ("vgg16", rt.MATH_BF16, 209, 97)])
def test_same_bits_in_pieces(binding, name, math, N, image):
    """An image's result does not depend on whether its batch was computed in pieces."""
    rt.set_math_mode(math)
    g = getattr(graphs, name)(batch=N, seed=1, image=image, **({"softmax": False} if name == "resnet50" else {}))
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    x = torch.from_numpy(rand(1, *g.input_shape)).pin_memory().numpy()
    outs, n0 = [], rt.form_counters()["in_pieces"]
    while rt.form_counters()["in_pieces"] < n0 + 3:
        outs.append(p.run(binding, x)[0])
        assert len(outs) < 24
    for y in outs[2:]:   # (the first pass runs unfused)
        assert np.array_equal(y, outs[1])
    assert rt.last_error() == 0


def test_pieces_take_the_forms_of_the_batch(binding):
    """Layers on 8x8 images, for which 450 of them share tiles and a piece's 80 to 150 by themselves would not: the two forms
    sum up in orders of their own, and an image has the same bits all the same."""
    rt.set_math_mode(rt.MATH_BF16)
    g = graphs.Graph((450, 3, 64, 64), seed=1)
    v = g.maxpool(g.relu(g.conv(0, *g.he_conv(64, 3, 7, 7), pads=(3, 3), strides=(2, 2))), (3, 3), (1, 1), (2, 2))
    v = g.relu(g.conv(v, *g.he_conv(128, 64, 1, 1), strides=(2, 2)))
    for _ in range(3):
        v = g.relu(g.conv(v, *g.he_conv(128, 128, 3, 3), pads=(1, 1)))
    g.mark_output(g.linear(g.flatten(g.gap(v)), 128, 40))
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    x = torch.from_numpy(rand(1, *g.input_shape)).pin_memory().numpy()
    outs, n0 = [], rt.form_counters()
    for _ in range(12):
        outs.append(p.run(binding, x)[0])
    n1 = rt.form_counters()
    assert n1["in_pieces"] > n0["in_pieces"] and n1["column_strips"] == n0["column_strips"]
    for y in outs[2:]:
        assert np.array_equal(y, outs[1])
    assert rt.last_error() == 0


def test_other_tensors_behind_pieces(native_libs):
    """A program that goes on like the recorded one until its result has been read, and then reads another tensor."""
    rt.set_math_mode(rt.MATH_BF16)
    N = 128
    run, want = small_model(N)
    x = torch.from_numpy(rand(10, N, 16, 96, 96)).pin_memory().numpy()
    logits, means = want(x)
    n0 = rt.form_counters()["in_pieces"]
    for i, mid in enumerate([False] * (PASSES + 2) + [True, False, True, False, False]):
        got = run(x, mid=mid)
        assert max_rel_err(got[0], logits) <= 2e-2, i
        if mid:
            assert max_rel_err(got[1], means) <= 2e-2, i
            assert i > PASSES + 2 or rt.form_counters()["in_pieces"] > n0 + 1
    assert rt.last_error() == 0


def test_memory_is_given_back(native_libs):
    """When an allocation fails, what batches in pieces work in makes room for it.  (In a process of its own, which
    would end at the failure.)"""
    code = """
import numpy as np, torch
import test_gpu_host_batches as t
from occamy_b200 import graphs, replay, runtime as rt
rt.set_math_mode(rt.MATH_BF16)
b = replay.Binding()
g = t.net(512, 224)
p = g.to_program()
p.lower(fuse=1)
x = torch.from_numpy(t.rand(1, *g.input_shape)).pin_memory().numpy()
for _ in range(t.PASSES + 3):
    (want,) = p.run(b, x)
assert rt.form_counters()["in_pieces"] > 0
free = torch.cuda.mem_get_info()[0]
keep = torch.empty(free - (96 << 20), dtype=torch.uint8, device="cuda")
buf = rt.DeviceBuffer(192 << 20)   # more than is left: the pieces' memory (some 500 MB) has to go
del keep
torch.cuda.empty_cache()
for _ in range(t.PASSES):
    (got,) = p.run(b, x)
    assert np.array_equal(got, want)
assert rt.last_error() == 0
"""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
