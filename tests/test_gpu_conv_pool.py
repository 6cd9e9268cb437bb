"""2x2 max pools taken along by the convolution in front of them, at ragged sizes and odd heights and widths,
against the CPU oracle and the same calls made apart."""
import numpy as np
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("fuse", [replay.FUSE_REFERENCE, replay.FUSE_NONE])
@pytest.mark.parametrize("N,C,H,W,K", [(8, 64, 112, 112, 64), (30, 64, 31, 45, 64), (5, 64, 57, 224, 64), (60, 64, 17, 15, 64),
                                       (24, 128, 56, 56, 256), (61, 256, 15, 29, 256), (90, 192, 14, 14, 512)])
def test_conv_pool(binding, N, C, H, W, K, fuse, mode):
    g = graphs.Graph((N, C, H, W), seed=N + C + H)
    v = g.relu(g.conv(0, *g.he_conv(K, C, 3, 3), pads=(1, 1)))
    v = g.maxpool(v, (2, 2), (0, 0), (2, 2))
    g.mark_output(v)
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=fuse)
    n0 = rt.form_counters()["pooled"]
    got = [p.run(binding, x)[0] for _ in range(4)]
    if fuse == replay.FUSE_REFERENCE:   # 64 channels: the strips, which are bf16 and not worth it on small images
        taken = K >= 256 or (mode == rt.MATH_BF16 and H > 17)
        assert (rt.form_counters()["pooled"] - n0 >= 3) == taken
    for y in got:
        assert max_rel_err(y, want) <= 2e-2
        if fuse == replay.FUSE_REFERENCE:   # the largest of rounded values is the rounded largest
            assert np.array_equal(y, got[0])
    assert rt.last_error() == 0
