"""Layers that the runtime holds back until the next one comes by (a block's last convolution, the first of two summands):
whatever happens in between, they have run by the time anybody can tell."""
import numpy as np
import pytest

from calls import Inference, rand
from helpers import max_rel_err
from occamy_b200 import runtime as rt
from oracle import ref

pytestmark = pytest.mark.gpu
PASSES = 7   # recorded, call by call, recorded as graphs, replayed


def test_stream_of_the_caller_is_behind_a_held_layer(native_libs):
    """A block's end waits for the 1x1 convolution behind it; who asks for the stream orders work behind both."""
    rt.set_math_mode(rt.MATH_BF16)
    x = rand(1, 3, 64, 9, 11)
    (wz, bz), (wa, ba) = [(rand(k, 128, 64, 1, 1, scale=0.1), rand(k + 1, 128)) for k in (2, 4)]
    wt, bt = rand(6, 64, 128, 1, 1, scale=0.1), rand(7, 64)
    y_want = np.maximum(ref.conv2d(x, wa, ba) + ref.conv2d(x, wz, bz, act=1), 0)
    t_want = ref.conv2d(y_want, wt, bt, act=1)
    for i in range(PASSES):
        with Inference() as f:
            px = f.put(x)
            z, o = f.conv(px, x.shape, f.put(wz), wz.shape, f.put(bz), act=1)
            a, _ = f.conv(px, x.shape, f.put(wa), wa.shape, f.put(ba), act=5)
            n0 = rt.counters()["tc_launches"]
            y = f.relu(f.op(0, a, o, z, o), o)
            rt.lib().occamy_stream()
            if i:   # (the first time through, the convolution was launched when it came by)
                assert rt.counters()["tc_launches"] == n0 + 1, i
            t, to = f.conv(y, o, f.put(wt), wt.shape, f.put(bt), act=1)
            t_got, y_got = f.get(t, to), f.get(y, o)
        assert max_rel_err(t_got, t_want) <= 2e-2 and max_rel_err(y_got, y_want) <= 2e-2, i
    assert rt.last_error() == 0
