"""Replayed inferences must compute from this inference's inputs and constants, whichever way those came in:
hand-made call sequences with a fresh input for every pass, against the CPU oracle."""
import numpy as np
import pytest
import torch

from calls import Inference, rand
from helpers import max_rel_err
from occamy_b200 import graphs
from occamy_b200 import runtime as rt
from oracle import ref

pytestmark = pytest.mark.gpu

PASSES = 10   # recorded, fused, quiet, captured once per pool block, then replayed


def device(a):
    t = torch.from_numpy(a).cuda()
    torch.cuda.synchronize()
    return t


# convolutions that the 16-bit path refuses: by their activation, their stride, their channels
@pytest.mark.parametrize("c,k,r,stride,act", [(16, 16, 3, 1, 0), (16, 16, 3, 1, 2), (3, 16, 11, 4, 1), (16, 16, 3, 3, 5),
                                              (20, 16, 3, 1, 1), (3, 12, 3, 1, 1)])
def test_device_input_of_a_refused_convolution(native_libs, c, k, r, stride, act):
    rt.set_math_mode(rt.MATH_BF16)
    w, b = rand(1, k, c, r, r, scale=0.2), rand(2, k)
    kept = []   # no address comes twice
    for i in range(PASSES):
        x = rand(100 + i, 2, c, 23, 21)
        kept.append(device(x))
        with Inference() as f:
            y, o = f.conv(f.copy(kept[-1].data_ptr(), x.nbytes), x.shape, f.put(w), w.shape, f.put(b), (1, 1),
                          (stride, stride), act=act)
            got = f.get(y, o)
        want = ref.conv2d(x, w, b, (1, 1), (stride, stride), act=act)
        assert max_rel_err(got, want) <= 2e-2, i
    assert rt.last_error() == 0


def test_constants_in_front_of_the_batch(native_libs):
    """Two sets of weights at addresses of their own, uploaded before the batch: each inference uses its own."""
    rt.set_math_mode(rt.MATH_BF16)
    sets = [[(rand(10 * s + i, 16, 16, 3, 3, scale=0.1), rand(50 + 10 * s + i, 16)) for i in range(3)] for s in (0, 1)]
    for i in range(4 * PASSES):
        layers = sets[(i * i // 3) % 2]
        x = want = rand(i, 2, 16, 12, 12)
        with Inference() as f:
            ws = [(f.put(w), f.put(b)) for w, b in layers]
            y = f.put(x)
            for (w, b), (pw, pb) in zip(layers, ws):
                y, o = f.conv(y, x.shape, pw, w.shape, pb, (1, 1), act=1)
                want = ref.conv2d(want, w, b, (1, 1), act=1)
            got = f.get(y, o)
        assert max_rel_err(got, want) <= 2e-2, i
    assert rt.last_error() == 0


def test_large_operand_changed_in_one_place(native_libs):
    """An operand of an element-wise call or a product may be an input: every byte of it counts."""
    rt.set_math_mode(rt.MATH_BF16)
    x, z, m = rand(1, 1, 64, 64, 64), rand(2, 1, 64, 64, 64), rand(3, 256, 512)
    a = rand(4, 8, 256)
    for i in range(PASSES):
        z.reshape(-1)[70001 + 4099 * i] += 3.0
        m.reshape(-1)[30001 + 4099 * i] += 3.0
        with Inference() as f:
            s = f.get(f.op(0, f.put(x), x.shape, f.put(z), z.shape), x.shape)
            y, o = f.matmul(f.put(a), a.shape, f.put(m), m.shape, trans_b=0)
            y = f.get(y, o)
        assert np.array_equal(s, x + z), i
        assert max_rel_err(y, ref.matmul2d(a, m)) <= 2e-2, i
    assert rt.last_error() == 0


def test_copies_from_tensors_outside_the_pool(native_libs):
    """The same calls but for which of two tensors of the runtime's, outside the pool, is copied in."""
    rt.set_math_mode(rt.MATH_BF16)
    x, w, b = rand(1, 1, 16, 12, 12), rand(2, 16, 16, 3, 3, scale=0.1), rand(3, 16)
    t, u = rt.DeviceBuffer(x.nbytes), rt.DeviceBuffer.from_numpy(rand(4, *x.shape))
    mid = ref.conv2d(x, w, b, (1, 1))
    for i, which in enumerate([u] * 4 + [t, u, t, t, u, t]):
        with Inference() as f:
            px, pw, pb = f.put(x), f.put(w), f.put(b)
            f.conv(px, x.shape, pw, w.shape, pb, (1, 1), act=5, y=t.ptr)
            r = f.relu(t.ptr, x.shape)
            got = f.get(f.copy(which.ptr, x.nbytes), x.shape), f.get(r, x.shape)
        if i == 4:   # leaves the recorded sequence behind a tensor that was skipped: reported, and recorded anew
            assert rt.last_error() == 990
            continue
        assert max_rel_err(got[0], mid if which is t else rand(4, *x.shape)) <= 2e-2
        assert max_rel_err(got[1], np.maximum(mid, 0)) <= 2e-2
        assert rt.last_error() == 0


@pytest.mark.parametrize("outside", [True, False])
def test_source_of_a_copy_is_overwritten(native_libs, outside):
    """What was copied in stays what it was, whatever happens to where it came from."""
    rt.set_math_mode(rt.MATH_BF16)
    w, b, z = rand(1, 16, 16, 3, 3, scale=0.1), rand(2, 16), rand(3, 1, 16, 12, 12)

    def run(x, conv):
        with Inference() as f:
            src, at = device(x), f.at
            s = f.place(x.nbytes)
            t = f.place(x.nbytes)
            rt.lib().wrapDNNMemcpy(s, src.data_ptr(), x.nbytes, 3, None)
            rt.lib().wrapDNNMemcpy(t, src.data_ptr() if outside else s, x.nbytes, 3, None)
            if outside:
                rt.synchronize()
                src.zero_()
                torch.cuda.synchronize()
            else:
                f.put(z, at=at)
            if conv:
                y, o = f.conv(t, x.shape, f.put(w), w.shape, f.put(b), (1, 1), act=5)
            else:
                y, o = f.relu(t, x.shape), x.shape
            return f.get(y, o)
    for i, conv in enumerate([True] * 7 + [False, True, False] + [True] * 4 + [False]):
        x = rand(20 + i, 1, 16, 12, 12)
        got = run(x, conv)
        if conv:
            assert max_rel_err(got, ref.conv2d(x, w, b, (1, 1))) <= 2e-2
        else:
            assert np.array_equal(got, np.maximum(x, 0))
    assert rt.last_error() == 0


def test_tensor_outside_the_pool_in_a_buffer_of_the_runtime(binding):
    """An in-place convolution by direct calls leaves its result in a buffer of the runtime's; a model that was
    captured while that buffer was free is replayed before the result is read."""
    rt.set_math_mode(rt.MATH_BF16)
    g = graphs.resnet50(batch=1, seed=1, softmax=False, image=64)
    p = g.to_program()
    p.lower(fuse=0)
    v = graphs.make_input(g, 1)
    for _ in range(PASSES):
        (want_model,) = p.run(binding, v)
    L, d = rt.lib(), rt.dims
    x, w = rand(1, 1, 64, 16, 16), rand(2, 64, 64, 1, 1, scale=0.2)
    t, tw = rt.DeviceBuffer.from_numpy(x), rt.DeviceBuffer.from_numpy(w)
    want = x
    for i in range(4):
        for _ in range(2):
            L.DNNConvFunc(None, t.ptr, d(x.shape), tw.ptr, d(w.shape), None, 0, 0, 1, d((0, 0)), d((1, 1)), t.ptr)
            want = ref.conv2d(want, w)
        (y,) = p.run(binding, v)
        assert np.array_equal(y, want_model)
        assert max_rel_err(t.to_numpy(x.shape), want) <= 5e-2, i
        want = t.to_numpy(x.shape)
    assert rt.last_error() == 0


def test_constants_at_one_address(native_libs):
    """A constant whose address was another one's for a while is found again: no upload in every inference."""
    rt.set_math_mode(rt.MATH_BF16)
    buf = rand(1, 64, 16, 3, 3, scale=0.1)
    x = rand(2, 1, 16, 12, 12)

    def run(k):
        w = buf[:k]   # the same address, another size
        with Inference() as f:
            n0 = rt.counters()["h2d_bytes"]
            y, o = f.conv(f.put(x), x.shape, f.put(w), w.shape, pads=(1, 1))
            got = f.get(y, o)
        assert max_rel_err(got, ref.conv2d(x, w, None, (1, 1))) <= 2e-2
        return rt.counters()["h2d_bytes"] - n0
    for k in [16] * 3 + [64] * 3 + [16]:
        run(k)
    assert [run(16) for _ in range(3)] == [x.nbytes] * 3
    assert rt.last_error() == 0
