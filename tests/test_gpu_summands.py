"""Sums of two convolutions in one kernel (a block's last convolution and its projection shortcut): odd sizes, strides on
either side, 3x3 against 1x1, channel counts with remainders, against the CPU oracle; and sums that are not taken."""
import numpy as np
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu
TOL = {rt.MATH_FP32: 1e-4, rt.MATH_BF16: 2e-2, rt.MATH_F16: 2e-2}


def _block(N, C, H, W, M, K, R, s_main, s_short, shortcut_first=False, act=True, relu_before=False, twice=False):
    """input -> 3x3 (M channels) -> conv a (R x R, K channels); input -> conv b (1x1, K channels); a + b."""
    g = graphs.Graph((N, C, H, W), seed=N + C + H + K)
    x = g.relu(g.conv(0, *g.he_conv(C, C, 1, 1)))
    t = g.relu(g.conv(x, *g.he_conv(M, C, 3, 3), pads=(1, 1), strides=(s_short // s_main,) * 2))

    def main():
        return g.conv(t, *g.he_conv(K, M, R, R), pads=(R // 2, R // 2), strides=(s_main, s_main))

    def short():
        return g.conv(x, *g.he_conv(K, C, 1, 1), strides=(s_short, s_short))

    a, b = (short(), main()) if shortcut_first else (main(), short())
    if relu_before:
        a = g.relu(a)
    y = g.add(a, b)
    if act:
        y = g.relu(y)
    if twice:   # the first summand has another reader
        y = g.add(y, a)
    g.mark_output(y)
    return g


def _run(binding, g, mode, fuse, taken):
    x = graphs.make_input(g, 3)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=fuse)
    n0 = rt.form_counters()["summed"]
    got = [p.run(binding, x)[0] for _ in range(4)]
    assert (rt.form_counters()["summed"] > n0) == taken
    for y in got:
        assert max_rel_err(y, want) <= TOL[mode]
    assert np.array_equal(got[2], got[3])
    assert rt.last_error() == 0


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("fuse", [replay.FUSE_REFERENCE, replay.FUSE_NONE])
@pytest.mark.parametrize("N,C,H,W,M,K,R,s_main,s_short", [
    (2, 64, 56, 56, 64, 256, 1, 1, 1),      # one row of pixels for both
    (61, 64, 51, 51, 64, 256, 1, 1, 1),     # several waves of tiles, nothing divides
    (3, 256, 29, 31, 128, 512, 1, 1, 2),    # strided shortcut, odd sizes
    (40, 256, 29, 31, 128, 512, 1, 1, 2),
    (1, 1024, 14, 14, 512, 2048, 1, 1, 2),  # clusters that share a reduction
    (64, 512, 13, 13, 256, 1024, 1, 1, 2),  # CTA pairs, an odd number of pixel tiles
    (33, 64, 28, 28, 128, 128, 3, 1, 2),    # 3x3 with a 1x1
    (5, 128, 17, 19, 64, 72, 3, 2, 2),      # both strided, channel tile with a remainder
])
def test_summands(binding, N, C, H, W, M, K, R, s_main, s_short, fuse, mode):
    _run(binding, _block(N, C, H, W, M, K, R, s_main, s_short), mode, fuse, True)


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_FP32])   # (fp32: apart, for the longer sum would cost digits)
@pytest.mark.parametrize("N,kw,taken", [(4, dict(shortcut_first=True), True), (6, dict(act=False), True),
                                        (8, dict(relu_before=True), False), (10, dict(twice=True), False)])
def test_summand_forms(binding, N, kw, taken, mode):
    # (batches of their own: what a recorded sequence skips stays skipped for another one that begins like it)
    _run(binding, _block(N + (mode == rt.MATH_FP32), 64, 21, 23, 64, 128, 1, 1, 1, **kw), mode, replay.FUSE_REFERENCE,
         taken and mode != rt.MATH_FP32)


def test_summands_of_unlike_steps_run_apart(binding):
    """96 channels go in steps of 32, 64 in steps of 64: no common ring."""
    _run(binding, _block(4, 96, 21, 23, 64, 128, 1, 1, 1), rt.MATH_BF16, replay.FUSE_REFERENCE, False)
