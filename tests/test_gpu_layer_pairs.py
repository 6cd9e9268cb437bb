"""A block's last convolution and the 1x1 convolution behind it as one kernel, both results kept: with a shortcut tensor and
with a projection (strided or not), image sizes that no tile divides, several chunks of channels, both 16-bit types; and
the same layers where there are too few pixels, or where the second layer is not of the kind.  Against the CPU oracle."""
import numpy as np
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


def _blocks(N, C, H, W, M, K1, K2, stride, window=1, relu=True):
    """Two blocks: the first ends in relu(1x1 conv of M channels + shortcut) with K1 channels, the second begins with a
    convolution to K2 channels and adds its end to the first one's result."""
    g = graphs.Graph((N, C, H, W), seed=N + C + H + K1)
    x = g.relu(g.conv(0, *g.he_conv(C, C, 1, 1)))
    t = g.relu(g.conv(x, *g.he_conv(M, C, 1, 1), strides=(stride, stride)))
    y = g.conv(t, *g.he_conv(K1, M, 1, 1))
    sc = g.conv(x, *g.he_conv(K1, C, 1, 1), strides=(stride, stride)) if C != K1 or stride != 1 else x
    y = g.relu(g.add(y, sc))
    r = g.conv(y, *g.he_conv(K2, K1, window, window), pads=(window // 2, window // 2))
    r = g.relu(r) if relu else r
    z = g.conv(r, *g.he_conv(K1, K2, 1, 1))
    g.mark_output(g.relu(g.add(z, y)))
    return g


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("fuse", [replay.FUSE_REFERENCE, replay.FUSE_NONE])
@pytest.mark.parametrize("N,C,H,W,M,K1,K2,stride,kw,taken", [
    (13, 256, 56, 56, 64, 256, 64, 1, {}, True),      # a shortcut tensor
    (61, 64, 26, 25, 64, 256, 64, 1, {}, True),       # a projection over the same pixels; nothing divides
    (53, 128, 55, 53, 128, 512, 128, 2, {}, True),    # a strided one: boxes of pixels, four blocks of x, four chunks
    (40, 128, 31, 33, 64, 128, 128, 1, {}, True),     # one chunk
    (49, 384, 28, 28, 192, 384, 64, 1, {}, True),     # an odd number of chunks
    (6, 256, 55, 57, 64, 256, 64, 1, {}, False),      # too few pixels
    (6, 256, 56, 57, 64, 256, 64, 1, {}, True),       # just enough
    (14, 256, 56, 56, 64, 256, 64, 1, dict(window=3), False),
    (15, 256, 56, 56, 64, 256, 64, 1, dict(relu=False), False),
    (16, 256, 56, 56, 64, 256, 72, 1, {}, False),
    (53, 256, 55, 53, 128, 512, 128, 2, {}, False),   # six blocks of x
])
def test_pairs(binding, N, C, H, W, M, K1, K2, stride, kw, taken, fuse, mode):
    g = _blocks(N, C, H, W, M, K1, K2, stride, **kw)
    x = graphs.make_input(g, 3)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=fuse)
    n0 = rt.form_counters()["pairs"]
    got = [p.run(binding, x)[0] for _ in range(4)]
    assert (rt.form_counters()["pairs"] > n0) == taken
    for y in got:
        assert max_rel_err(y, want) <= 2e-2
    assert np.array_equal(got[2], got[3])
    assert rt.last_error() == 0


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("act", ["relu", "clip"])
@pytest.mark.parametrize("N,C,H,W,M,K1,K2", [(3, 64, 19, 23, 64, 128, 64), (61, 64, 26, 25, 64, 256, 64), (9, 32, 25, 28, 128, 256, 256)])
def test_first_result_that_is_read_once(binding, N, C, H, W, M, K1, K2, act, mode):
    """Nobody but the second layer reads the first one's result, whose memory is handed out again while that layer's bias and
    activation, calls of their own, are still to come: they are part of it all the same, with the bits of the fused call."""
    g = graphs.Graph((N, C, H, W), seed=N + K1)
    x = g.relu(g.conv(0, *g.he_conv(C, C, 1, 1)))
    t = g.relu(g.conv(x, *g.he_conv(M, C, 3, 3), pads=(1, 1)))
    y = g.relu(g.add(g.conv(t, *g.he_conv(K1, M, 1, 1)), g.conv(x, *g.he_conv(K1, C, 1, 1))))
    r = g.conv(y, *g.he_conv(K2, K1, 1, 1))
    r = g.relu(r) if act == "relu" else g.clip(r, 0.0, 6.0)
    for _ in range(2):
        r = g.relu(g.conv(r, *g.he_conv(K2, K2, 3, 3), pads=(1, 1)))
    g.mark_output(r)
    x = graphs.make_input(g, 3)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    got, launches = [], []
    for fuse in (replay.FUSE_WITH_CLIP, replay.FUSE_NONE):
        p = g.to_program()
        p.lower(fuse=fuse)
        for _ in range(4):
            n0 = rt.counters()["launches"]
            y = p.run(binding, x)[0]
            n = rt.counters()["launches"] - n0
        got.append(y)
        launches.append(n)
        assert max_rel_err(y, want) <= 2e-2
    assert np.array_equal(got[0], got[1])
    assert launches[1] <= launches[0] + 1   # (one more where the pair is one kernel in the first)
    assert rt.last_error() == 0
