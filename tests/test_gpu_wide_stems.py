"""RGB stems with filters wider than seven columns and the max pool behind them: windows written out in 128-byte rows (of
images so narrow that an MMA reads far beyond a row, and wider ones), and windows read in place, where shared memory does
not suffice for the other form.  Odd sizes, several bands, more of them than SMs."""
import ctypes as C

import numpy as np
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt
from oracle import ref
from test_stem_layout import Layout, row_bytes

pytestmark = pytest.mark.gpu


def _form(R, S, W, pad):
    fn = getattr(C.CDLL(rt.LIB_PATH), "_ZN3occ16stem_pool_layoutEiiiiibPNS_14StemPoolLayoutE")
    fn.restype, fn.argtypes = C.c_bool, [C.c_int] * 5 + [C.c_bool, C.POINTER(Layout)]
    m, taps = Layout(), (S + 3) // 4 * 4
    Q = (W + 2 * pad - S) // 2 + 1
    pitch = max(row_bytes(taps, 2, 4, Q), (W + pad + 7) // 8 * 8 * 8)
    assert fn(R, taps * 4, 2, Q, pitch, True, m)
    return m.tiled, m.bk if m.tiled else 0


@pytest.mark.parametrize("act", ["relu", "clip"])
@pytest.mark.parametrize("N,H,W,R,S,pad,form", [
    (2, 41, 44, 9, 9, 4, (1, 64)),         # 22 columns of 128
    (3, 30, 12, 11, 11, 5, (1, 64)),       # 6
    (5, 33, 40, 7, 15, 3, (1, 64)),        # 64 values to a window
    (170, 51, 70, 9, 9, 4, (1, 64)),
    (2, 61, 121, 11, 11, 5, (0, 0)),
    (2, 45, 226, 11, 13, 5, (0, 0)),       # 64 values
    (170, 35, 231, 9, 9, 4, (0, 0)),       # 116 columns, bands of several images to an SM
    (1, 224, 224, 11, 11, 5, (0, 0)),
    (2, 10, 200, 9, 9, 4, (0, 0)),         # every row of the output reaches over an edge
])
def test_wide_stem_with_max_pool(binding, N, H, W, R, S, pad, form, act):
    g = graphs.Graph((N, 3, H, W), seed=N + H + W)
    w, b = g.he_conv(64, 3, R, S)
    y = g.conv(0, w, b, pads=(pad, pad), strides=(2, 2))
    y = g.relu(y) if act == "relu" else g.clip(y, -0.25, 0.75)
    g.mark_output(g.maxpool(y, (3, 3), (1, 1), (2, 2)))
    assert _form(R, S, W, pad) == form
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(rt.MATH_BF16)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    (apart,) = p.run(binding, x)            # convolution and pool one after the other
    n0 = rt.lib().occamy_fused_chains()
    (got,) = p.run(binding, x)
    assert rt.lib().occamy_fused_chains() == n0 + 1
    # Both factors of a product and the sum are rounded to bf16, 2^-8 of themselves each time; the clamp and the largest of
    # a window's values make no difference larger.
    most = ref.conv2d(np.abs(x), np.abs(w), np.abs(b), (pad, pad), (2, 2))
    bound = 1.02 * 3 * 2.0 ** -8 * ref.pool2d(most, (3, 3), (1, 1), (2, 2))
    for y in (apart, got):
        assert np.all(np.abs(y - want) <= bound)
        if act == "relu":
            assert max_rel_err(y, want) <= 2e-2
    assert np.array_equal(got, apart)       # rounded the same way, and the largest of the same values
    assert rt.last_error() == 0


def test_a_launch_that_was_made_before_encodes_nothing(binding):
    """Call by call (while launches are timed nothing is replayed), the tensor maps of a stem are those of the call before."""
    rt.set_math_mode(rt.MATH_BF16)
    g = graphs.Graph((2, 3, 60, 66), seed=5)
    y = g.relu(g.conv(0, *g.he_conv(64, 3, 7, 7), pads=(3, 3), strides=(2, 2)))
    g.mark_output(g.maxpool(y, (3, 3), (1, 1), (2, 2)))
    x = graphs.make_input(g, 1)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    rt.lib().occamy_profile_begin()
    encodes = []
    for _ in range(8):   # (two pool blocks in turn)
        p.run(binding, x)
        encodes.append(rt.counters()["tmap_encodes"])
    ms = (C.c_float * 64)()
    assert rt.lib().occamy_profile_end(ms, 64) >= 8
    assert encodes[4] == encodes[7], encodes


@pytest.mark.parametrize("R,pad", [(3, 3), (3, 5), (5, 5), (5, 4)])
def test_rows_of_padding_alone(binding, R, pad):
    """Padding as high as the filter: the first and last rows of the output are the bias."""
    rt.set_math_mode(rt.MATH_BF16)
    g = graphs.Graph((3, 3, 21, 26), seed=R + pad)
    y = g.relu(g.conv(0, *g.he_conv(64, 3, R, R), pads=(pad, pad), strides=(2, 2)))
    g.mark_output(g.maxpool(y, (3, 3), (1, 1), (2, 2)))
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    for _ in range(4):
        (got,) = p.run(binding, x)
        assert max_rel_err(got, want) <= 2e-2
    assert rt.last_error() == 0
