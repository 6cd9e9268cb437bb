"""Few-channel convolutions whose input rows are copied as they lie and read as overlapping windows: rows of more than one
tile, widths that nothing divides, one to four channels, strides, row taps outside the image, clamps, both 16-bit types.
Inputs and filters are numbers of the type, so that only the result is rounded: half a step of its last bit, 2^-8 of a
value in bf16 and 2^-11 in fp16."""
import numpy as np
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


def _round(a, mode):
    if mode == rt.MATH_F16:
        return np.asarray(a, np.float16).astype(np.float32)
    u = np.ascontiguousarray(a, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


def _run(binding, N, C, H, W, K, R, pad, stride, act, mode):
    g = graphs.Graph((N, C, H, W), seed=N + C + H)
    w, b = g.he_conv(K, C, R, R)
    v = g.conv(0, _round(w, mode), b, pads=(pad, pad), strides=(stride, stride))
    g.mark_output(g.relu(v) if act == "relu" else g.clip(v, -0.5, 0.75) if act == "clip" else v)
    x = _round(graphs.make_input(g, 1), mode)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    n0 = rt.form_counters()["input_rows"]
    got = [p.run(binding, x)[0] for _ in range(3)]   # (the first call by call: bias and clamp round again)
    assert max_rel_err(got[2], want) <= (2.0 ** -8 if mode == rt.MATH_BF16 else 2.0 ** -11) * 1.05
    assert np.array_equal(got[1], got[2])
    assert rt.last_error() == 0
    return rt.form_counters()["input_rows"] - n0


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("N,C,H,W,K,R,pad,stride,act", [
    (8, 3, 224, 224, 64, 3, 1, 1, "relu"),
    (20, 3, 97, 131, 64, 3, 1, 1, "relu"),     # two tiles to a row, neither whole
    (9, 3, 60, 300, 40, 3, 1, 1, "clip"),      # three; channels with a remainder
    (30, 3, 160, 112, 32, 3, 1, 2, "clip"),    # the shortest rows that are read this way
    (30, 3, 91, 56, 32, 3, 1, 1, "clip"),
    (12, 4, 222, 171, 24, 3, 1, 2, None),
    (7, 1, 150, 129, 64, 3, 2, 1, "relu"),     # a row of padding beyond the filter's reach into the image
    (40, 2, 120, 69, 16, 2, 0, 1, "relu"),
    (24, 3, 128, 128, 64, 1, 0, 1, "relu"),
])
def test_rows(binding, N, C, H, W, K, R, pad, stride, act, mode):
    assert _run(binding, N, C, H, W, K, R, pad, stride, act, mode) == 3


@pytest.mark.parametrize("N,C,H,W,K,R,pad,stride", [
    (8, 3, 120, 130, 64, 5, 2, 1),     # more rows of the filter
    (8, 3, 120, 130, 72, 3, 1, 1),     # ... channels of the result
    (8, 9, 120, 130, 64, 3, 1, 1),     # ... of the input
    (8, 3, 120, 130, 64, 3, 3, 1),     # padding as high as the filter
    (30, 3, 160, 97, 32, 3, 1, 2),     # short rows
    (40, 2, 120, 64, 16, 2, 0, 1),
    (24, 3, 97, 79, 64, 1, 0, 1),
])
def test_other_stems_read_windows(binding, N, C, H, W, K, R, pad, stride):
    assert _run(binding, N, C, H, W, K, R, pad, stride, "relu", rt.MATH_BF16) == 0
