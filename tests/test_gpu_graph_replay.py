"""Recorded inferences that run as CUDA graphs: same bits as call by call, and every way out of one
(another constant, another continuation, a wait or the end in the middle)."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from calls import Inference, rand
from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt
from oracle import ref

pytestmark = pytest.mark.gpu

PASSES = 9   # recorded, fused, quiet, captured once per pool block, then replayed


def _model(name, math, fuse, batch=2):
    rt.set_math_mode(math)
    kw = {"softmax": True} if name == "resnet50" else {}
    g = getattr(graphs, name)(batch=batch, seed=3, image=64, **kw)
    p = g.to_program()
    p.lower(fuse=fuse)
    return g, p


@pytest.mark.parametrize("io", ["host", "device"])
@pytest.mark.parametrize("name,math,fuse", [
    ("resnet50", rt.MATH_BF16, 1), ("resnet50", rt.MATH_BF16, 0), ("resnet50", rt.MATH_FP32, 1),
    ("mobilenet_v2", rt.MATH_F16, 1), ("vgg16", rt.MATH_BF16, 1)])
def test_same_bits_and_launches(binding, name, math, fuse, io):
    g, p = _model(name, math, fuse)
    xs = [graphs.make_input(g, s) for s in (1, 2)]
    dev = [torch.from_numpy(x).cuda() for x in xs]
    outs, launches = [], []
    for i in range(PASSES):
        n0 = rt.counters()["launches"]
        if io == "host":
            (y,) = p.run(binding, xs[i % 2])
        else:
            yd = torch.empty(g.shapes[g.outputs[0]], device="cuda")
            torch.cuda.synchronize()
            p.run_raw(binding, dev[i % 2].data_ptr(), 3, [yd.data_ptr()], 3)
            rt.synchronize()
            y = yd.cpu().numpy()
        outs.append(y)
        launches.append(rt.counters()["launches"] - n0)
    assert rt.last_error() == 0
    for i in range(3, PASSES):   # pass 2 ran call by call with the chains of pass 1
        assert np.array_equal(outs[i], outs[i - 2])
    assert len(set(launches[3:])) == 1
    (want,) = run_graph_oracle(g, xs[0])
    assert max_rel_err(outs[-1 if PASSES % 2 else -2], want) <= (1e-4 if math == rt.MATH_FP32 else 3e-2)


def test_changed_constant_is_seen(binding):
    g, p = _model("vgg16", rt.MATH_BF16, 1)
    x = graphs.make_input(g, 1)
    conv = [n for n in g.nodes if n.op == "conv"][5]
    w = next(a for a in p._keep if a.shape == g.consts[conv.ins[1]].shape and np.array_equal(a, g.consts[conv.ins[1]]))
    for _ in range(PASSES):
        (before,) = p.run(binding, x)
    old = w.copy()
    for scale in (1.5, 0.5, 1.0):   # there and back again
        w[...] = old * scale
        g.consts[conv.ins[1]] = w
        (want,) = run_graph_oracle(g, x)
        for _ in range(PASSES):
            (y,) = p.run(binding, x)
            assert max_rel_err(y, want) <= 3e-2
    assert np.array_equal(y, before)
    assert rt.last_error() == 0


def test_two_sets_of_weights(binding):
    """One architecture, two models served in turn: same calls, other constants."""
    rt.set_math_mode(rt.MATH_BF16)
    models = []
    for seed in (1, 2):
        g = graphs.resnet50(batch=1, seed=seed, image=64, softmax=False)
        p = g.to_program()
        p.lower(fuse=1)
        x = graphs.make_input(g, seed)
        models.append((p, x, run_graph_oracle(g, x)[0]))
    for i in range(4 * PASSES):
        p, x, want = models[(i * i // 3) % 2]
        (y,) = p.run(binding, x)
        assert max_rel_err(y, want) <= 2e-2
    assert rt.last_error() == 0


def test_other_continuation(binding):
    """Two models with the same first layers: the recorded one is left in the middle of its window."""
    rt.set_math_mode(rt.MATH_F16)   # 18 layers: bf16 storage alone is off by 5e-2
    models = []
    for tail in ("relu", "clip", "add"):
        g = graphs.Graph((2, 16, 20, 20), seed=5)
        y = 0
        for _ in range(18):
            w, b = g.he_conv(16, 16, 3, 3)
            y = g.relu(g.conv(y, w, b, pads=(1, 1)))
        y = g.relu(y) if tail == "relu" else g.clip(y, 0.0, 0.7) if tail == "clip" else g.add(y, y)
        g.mark_output(y)
        p = g.to_program()
        p.lower(fuse=1)
        x = graphs.make_input(g, 4)
        models.append((p, x, run_graph_oracle(g, x)[0]))
    for which in [0] * PASSES + [1, 0, 1, 0, 0] + [1] * PASSES + [2, 0, 1, 2, 2, 1, 0]:
        p, x, want = models[which]
        (y,) = p.run(binding, x)
        assert max_rel_err(y, want) <= 2e-2
    assert rt.last_error() == 0


class _HandModel:
    """x -> conv -> conv -> ... by direct ABI calls, so that a test can stop in the middle."""

    def __init__(self, layers=20, c=16, hw=12):
        r = np.random.default_rng(0)
        self.n, self.shape = layers, (1, c, hw, hw)
        self.w = [(r.standard_normal((c, c, 3, 3)) * 0.08).astype(np.float32) for _ in range(layers)]
        self.b = [(r.standard_normal(c) * 0.1).astype(np.float32) for _ in range(layers)]
        self.x = r.standard_normal(self.shape).astype(np.float32)

    def run(self, upto=None, between=None, read_at=None):
        L = rt.lib()
        h, pool, out = C.c_void_p(), C.c_void_p(), None
        L.cudnnCreate(C.byref(h))
        L.wrapDNNMemPoolInit(C.byref(pool), 1 << 22)
        at = 0

        def place(nbytes):
            nonlocal at
            p = C.c_void_p()
            L.wrapDNNMemOffset(C.byref(p), pool, at, nbytes)
            at += (nbytes + 31) // 32 * 32
            return p.value
        cur = place(self.x.nbytes)
        L.wrapDNNMemcpy(cur, self.x.ctypes.data, self.x.nbytes, 1, None)
        res = []
        for i in range(self.n if upto is None else upto):
            w, b = place(self.w[i].nbytes), place(self.b[i].nbytes)
            L.wrapDNNMemcpy(w, self.w[i].ctypes.data, self.w[i].nbytes, 1, None)
            L.wrapDNNMemcpy(b, self.b[i].ctypes.data, self.b[i].nbytes, 1, None)
            y = place(self.x.nbytes)
            L.DNNConvBiasActivFunc(h, cur, rt.dims(self.shape), w, rt.dims(self.w[i].shape), b,
                                   rt.dims((1, self.shape[1], 1, 1)), None, 0, 0, rt.dims((1, 1)),
                                   rt.dims((1, 1)), 1, y)
            cur = y
            if between is not None and i == between[0]:
                between[1]()
            if read_at == i:
                mid = np.empty(self.shape, np.float32)
                L.wrapDNNMemcpy(mid.ctypes.data, cur, mid.nbytes, 2, None)
                res.append(mid)
        out = np.empty(self.shape, np.float32)
        L.wrapDNNMemcpy(out.ctypes.data, cur, out.nbytes, 2, None)
        L.wrapDNNDealloc(pool)
        L.cudnnDestroy(h)
        return [out] + res


def test_ways_out_of_the_middle(native_libs):
    rt.set_math_mode(rt.MATH_BF16)
    m = _HandModel()
    (want,) = m.run()
    for i in (3, 14, 19):
        full = {}
        for _ in range(PASSES):
            (y,) = m.run()
            assert np.array_equal(y, want)
        # a wait, a question for the stream, a read of an intermediate, an early end
        (y,) = m.run(between=(i, lambda: rt.synchronize()))
        assert np.array_equal(y, want)
        (y,) = m.run(between=(i, lambda: rt.lib().occamy_stream()))
        assert np.array_equal(y, want)
        y, mid = m.run(read_at=i)
        assert np.array_equal(y, want)
        (early,) = m.run(upto=i + 1)
        assert np.array_equal(early, mid)
        (y,) = m.run()
        assert np.array_equal(y, want)
    assert rt.last_error() == 0


@pytest.mark.parametrize("c", [3, 16])
def test_device_input_in_convolution_form(native_libs, c):
    """A batch copied in on the device arrives in the form its convolution takes; a program with the same
    beginning that reads it otherwise still sees the plain fp32 values."""
    rt.set_math_mode(rt.MATH_BF16)
    L = rt.lib()
    r = np.random.default_rng(1)
    w = (r.standard_normal((16, c, 3, 3)) * 0.2).astype(np.float32)
    b = r.standard_normal(16).astype(np.float32)
    from oracle import ref

    def infer(x, conv):
        xd = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        h, pool = C.c_void_p(), C.c_void_p()
        L.cudnnCreate(C.byref(h))
        L.wrapDNNMemPoolInit(C.byref(pool), 1 << 20)
        offs, at = [], 0
        for n in (x.nbytes, w.nbytes, b.nbytes, x.shape[0] * 16 * x.shape[2] * x.shape[3] * 4):
            offs.append(at)
            at += (n + 31) // 32 * 32

        def place(i, n):
            p = C.c_void_p()
            L.wrapDNNMemOffset(C.byref(p), pool, offs[i], n)
            return p.value
        px = place(0, x.nbytes)
        L.wrapDNNMemcpy(px, xd.data_ptr(), x.nbytes, 3, None)
        oshape = (x.shape[0], 16) + x.shape[2:] if conv else x.shape
        if conv:
            pw, pb = place(1, w.nbytes), place(2, b.nbytes)
            L.wrapDNNMemcpy(pw, w.ctypes.data, w.nbytes, 1, None)
            L.wrapDNNMemcpy(pb, b.ctypes.data, b.nbytes, 1, None)
            py = place(3, int(np.prod(oshape)) * 4)
            L.DNNConvBiasActivFunc(h, px, rt.dims(x.shape), pw, rt.dims(w.shape), pb, rt.dims((1, 16, 1, 1)), None,
                                   0, 0, rt.dims((1, 1)), rt.dims((1, 1)), 5, py)
        else:
            py = place(3, x.nbytes)
            L.DNNActiveFunc(h, px, rt.dims(x.shape), 1, py)
        out = np.empty(oshape, np.float32)
        L.wrapDNNMemcpy(out.ctypes.data, py, out.nbytes, 2, None)
        L.wrapDNNDealloc(pool)
        L.cudnnDestroy(h)
        return out

    for conv in [True] * 6 + [False, True, False] + [False] * 6 + [True, False]:
        x = r.standard_normal((2, c, 9, 11)).astype(np.float32)
        y = infer(x, conv)
        if conv:
            assert max_rel_err(y, ref.conv2d(x, w, b, (1, 1))) <= 2e-2
        else:
            assert np.array_equal(y, np.maximum(x, 0))
    assert rt.last_error() == 0


def test_wait_for_the_device_while_recording(native_libs):
    """A wait for the device, of whatever thread, neither fails nor costs a result while a graph is put together."""
    rt.set_math_mode(rt.MATH_BF16)
    m = _HandModel(layers=23)
    (want,) = m.run()

    def wait():
        t = threading.Thread(target=torch.cuda.synchronize)
        t.start()
        t.join()
        torch.cuda.synchronize()
    for i in (2, 15, 22):
        rt.lib().occamy_set_cross_call_fusion(0)   # forgets what was recorded
        rt.lib().occamy_set_cross_call_fusion(1)
        for _ in range(PASSES):
            (y,) = m.run(between=(i, wait))
            assert np.array_equal(y, want)
    assert rt.last_error() == 0


def test_graphs_out_of_use_are_destroyed(binding):
    """Weights that change again and again: the graphs that refer to the old ones are given back."""
    g, p = _model("resnet50", rt.MATH_BF16, 1, batch=1)
    x = graphs.make_input(g, 1)
    w = next(a for a in p._keep if a.size > 100000)
    free = []
    for i in range(120):
        w *= 1.0 + 1e-3 * (1 if i % 2 else -1)
        for _ in range(6):   # one pass notices, the next two are captured (one per pool block)
            p.run(binding, x)
        rt.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[39] - free[-1] <= 4 << 20, free[::10]
    assert rt.last_error() == 0


def test_call_with_many_dimensions(native_libs):
    """A call with more dimensions than a recorded call keeps, in the middle of an inference that is left early."""
    rt.set_math_mode(rt.MATH_BF16)
    shape, w, b = (1, 16, 12, 12), rand(1, 16, 16, 3, 3, scale=0.1), rand(2, 16)
    x = rand(3, *shape)

    def run(early):
        with Inference() as f:
            y, want = f.put(x), x
            pw, pb = f.put(w), f.put(b)
            for i in range(6):
                y, _ = f.conv(y, shape, pw, w.shape, pb, (1, 1), act=1)
                want = ref.conv2d(want, w, b, (1, 1), act=1)
                if i == 2:
                    z = f.place(x.nbytes)
                    f.L.CUDAClipFunc(y, z, rt.dims((1,) * 24 + (16, 144)), 0.0, 1.0, 26)
                    y, want = z, np.clip(want, 0.0, 1.0)
                if early and i == 4:
                    break
            return max_rel_err(f.get(y, shape), want)
    for early in [False] * PASSES + [True, False] * 4:
        assert run(early) <= 2e-2
    assert rt.last_error() == 0
