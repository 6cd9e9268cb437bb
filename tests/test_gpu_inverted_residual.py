"""The inverted-residual kernel (1x1 -> 3x3 depthwise -> 1x1 as one launch) at the edges of its tiles, chunks
and clusters, against the CPU oracle."""
import numpy as np
import pytest

from calls import Inference, rand
from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt
from oracle import ref

pytestmark = pytest.mark.gpu

# (N, C, H, W, E, K, stride): channels that are no multiple of a chunk or of the MMA's 16; one tile and many;
# ragged tiles; reductions in one to three input tiles; chunks shared by 1 to 8 CTAs
SHAPES = [
    (1, 16, 13, 9, 96, 24, 2),
    (2, 24, 20, 28, 144, 24, 1),
    (1, 24, 15, 17, 144, 32, 2),
    (3, 32, 28, 28, 192, 32, 1),
    (1, 64, 14, 14, 384, 96, 1),
    (3, 96, 14, 11, 576, 160, 2),
    (1, 160, 7, 7, 960, 160, 1),
    (40, 160, 7, 7, 960, 160, 1),
    (2, 40, 5, 3, 48, 8, 1),
    (30, 16, 60, 60, 96, 24, 2),
]


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("fuse", [replay.FUSE_REFERENCE, replay.FUSE_NONE])
@pytest.mark.parametrize("shape", SHAPES)
def test_block(binding, shape, fuse, mode):
    N, C, H, W, E, K, st = shape
    g = graphs.Graph((N, C, H, W), seed=sum(shape))
    x = g.clip(g.conv(0, *g.he_conv(C, C, 1, 1)), 0.0, 6.0)
    y = g.clip(g.conv(x, *g.he_conv(E, C, 1, 1)), 0.0, 6.0)
    y = g.clip(g.conv(y, *g.he_conv(E, 1, 3, 3), groups=E, pads=(1, 1), strides=(st, st)), 0.0, 6.0)
    y = g.conv(y, *g.he_conv(K, E, 1, 1))
    if st == 1 and K == C:
        y = g.add(x, y)
    g.mark_output(y)
    v = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, v)
    rt.set_math_mode(mode)
    rt.lib().occamy_set_cross_call_fusion(0)   # forgets what was recorded
    rt.lib().occamy_set_cross_call_fusion(1)
    p = g.to_program()
    p.lower(fuse=fuse)
    launches, forms = [], rt.form_counters()["inverted_residual"]
    for _ in range(4):
        before = rt.counters()["launches"]
        (got,) = p.run(binding, v)
        launches.append(rt.counters()["launches"] - before)
        assert max_rel_err(got, want) <= 2e-2
    assert launches[2] < launches[0]
    # large batches of small images run faster apart, and so does the last shape where the depthwise sums are fp32
    apart = shape == SHAPES[7] or (shape == SHAPES[9] and mode == rt.MATH_BF16)
    assert rt.form_counters()["inverted_residual"] - forms == (0 if apart else 3)
    assert rt.last_error() == 0


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("filters", ["no cache", "from the device", "from the host"])
def test_block_with_filters_that_do_not_stay(native_libs, filters, mode):
    """Filters without a resident packed copy: each of the three convolutions still gets its own."""
    rt.set_math_mode(mode)
    shape, E, K = (1, 16, 14, 14), 96, 24
    ws = [rand(1, 16, 16, 1, 1, scale=0.3), rand(2, E, 16, 1, 1, scale=0.3), rand(3, E, 1, 3, 3, scale=0.3),
          rand(4, K, E, 1, 1, scale=0.1)]
    dev = [rt.DeviceBuffer.from_numpy(w) for w in ws]
    groups = (1, 1, E, 1)
    rt.lib().occamy_set_weight_cache(0 if filters == "no cache" else 1)
    try:
        for i in range(6):
            x = rand(10 + i, *shape)
            with Inference() as f:
                y, o, want = f.put(x), shape, x
                for w, d, n in zip(ws, dev, groups):
                    pw = f.copy(d.ptr, w.nbytes) if filters == "from the device" else f.put(w)
                    pads = (w.shape[2] // 2,) * 2
                    y, o = f.conv(y, o, pw, w.shape, pads=pads, groups=n)
                    want = ref.conv2d(want, w, None, pads, groups=n)
                    if w is not ws[-1]:
                        y, want = f.clip(y, o, 0.0, 6.0), ref.clip(want, 0.0, 6.0)
                got = f.get(y, o)
            assert max_rel_err(got, want) <= 2e-2, i
    finally:
        rt.lib().occamy_set_weight_cache(1)
    assert rt.last_error() == 0


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("act", ["none", "relu", "clip"])
@pytest.mark.parametrize("N,C,H,E,K", [(1, 16, 14, 48, 24), (1, 24, 14, 144, 24), (40, 16, 28, 48, 16), (1, 64, 14, 96, 64),
                                       (1, 16, 14, 80, 24)])
def test_last_chunk(binding, N, C, H, E, K, act, mode):
    """Channels of the last chunk that do not exist count as zero, whatever an earlier kernel left in shared memory:
    NaN here.  (A clamp of the depthwise results would hide it.)"""
    g = graphs.Graph((N, C, H, H), seed=E + C)

    def end(v):
        return v if act == "none" else g.relu(v) if act == "relu" else g.clip(v, 0.0, 6.0)

    x = g.conv(0, *g.he_conv(C, C, 1, 1))
    y = end(g.conv(x, *g.he_conv(E, C, 1, 1)))
    y = end(g.conv(y, *g.he_conv(E, 1, 3, 3), groups=E, pads=(1, 1)))
    g.mark_output(g.conv(y, *g.he_conv(K, E, 1, 1)))
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    v = graphs.make_input(g, 1)
    bad = np.full_like(v, np.nan)
    (want,) = run_graph_oracle(g, v)
    forms = rt.form_counters()["inverted_residual"]
    for i in range(6):
        p.run(binding, bad)   # leaves NaN in every shared memory
        (got,) = p.run(binding, v)
        assert max_rel_err(got, want) <= 2e-2, i
    assert rt.form_counters()["inverted_residual"] >= forms + 10
    assert rt.last_error() == 0


@pytest.mark.parametrize("act", ["relu", "none"])
def test_overflow_of_the_depthwise_sums(binding, act):
    """fp16 sums that overflow in both directions are NaN, not a bound.  (A clip, by the ABI, makes a bound of NaN.)"""
    N, C, E, H = 1, 16, 96, 14
    g = graphs.Graph((N, C, H, H), seed=1)
    wx, bx = g.he_conv(C, C, 1, 1)
    x = g.conv(0, wx, bx)
    w1, b1 = np.zeros((E, C, 1, 1), np.float32), np.full(E, 6e4, np.float32)
    dw = np.zeros((E, 1, 3, 3), np.float32)
    dw[:, 0, 0], dw[:, 0, 2] = 6e4, -6e4     # +inf from the row above, -inf from the row below
    y = g.relu(g.conv(x, w1, b1))
    y = g.conv(y, dw, np.zeros(E, np.float32), groups=E, pads=(1, 1))
    y = g.relu(y) if act == "relu" else y
    g.mark_output(g.conv(y, *g.he_conv(24, E, 1, 1)))
    rt.set_math_mode(rt.MATH_F16)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    v = graphs.make_input(g, 1)
    forms = rt.form_counters()["inverted_residual"]
    for i in range(4):   # the first runs convolution by convolution
        (got,) = p.run(binding, v)
        assert np.isnan(got[:, :, 1:-1]).all(), i
    assert rt.form_counters()["inverted_residual"] >= forms + 3
    assert rt.last_error() == 0


@pytest.mark.parametrize("hi,sums_in_half", [(6.1, False), (6.0, True)])
def test_precision_of_the_depthwise_sums(binding, hi, sums_in_half):
    """2048 + 1 - 2048: 1 in fp32, 0 in fp16.  In the fp16 mode the depthwise kernel whose clamp has a bound that fp16
    does not hold (6.1) sums in fp32, and a block with one must not do otherwise.  (The first pass clamps apart.)"""
    N, C, E, K, H = 1, 16, 96, 24, 14
    g = graphs.Graph((N, C, H, H), seed=1)
    dw = np.zeros((E, 1, 3, 3), np.float32)
    dw[:, 0, 0, 0], dw[:, 0, 1, 1], dw[:, 0, 2, 2] = 2048.0, 1.0, -2048.0
    x = g.conv(0, *g.he_conv(C, C, 1, 1))
    y = g.clip(g.conv(x, np.zeros((E, C, 1, 1), np.float32), np.ones(E, np.float32)), 0.0, 6.0)
    y = g.clip(g.conv(y, dw, np.zeros(E, np.float32), groups=E, pads=(1, 1)), 0.0, hi)
    g.mark_output(g.conv(y, np.full((K, E, 1, 1), 0.125, np.float32), np.zeros(K, np.float32)))
    rt.set_math_mode(rt.MATH_F16)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    v = graphs.make_input(g, 1)
    forms = rt.form_counters()["inverted_residual"]
    for i in range(4):
        (got,) = p.run(binding, v)
        assert i == 0 or (got[:, :, 1:-1, 1:-1] == (0.0 if sums_in_half else E / 8)).all(), i
    assert (rt.form_counters()["inverted_residual"] > forms) == sums_in_half
    assert rt.last_error() == 0
