"""Few-channel convolutions with 64 output channels, whose kernel runs twice on an SM, at ragged sizes, against
the CPU oracle."""
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("clip", [False, True])
@pytest.mark.parametrize("N,C,H,W,K,R,stride", [(16, 3, 112, 112, 64, 3, 1), (9, 3, 97, 131, 64, 7, 2), (40, 5, 40, 57, 48, 5, 1),
                                                (33, 12, 33, 64, 64, 3, 2), (3, 1, 224, 200, 56, 3, 1)])
def test_stem(binding, N, C, H, W, K, R, stride, clip, mode):
    g = graphs.Graph((N, C, H, W), seed=N + C + H)
    y = g.conv(0, *g.he_conv(K, C, R, R), pads=(R // 2, R // 2), strides=(stride, stride))
    g.mark_output(g.clip(y, 0.0, 6.0) if clip else g.relu(y))
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    for _ in range(3):
        (got,) = p.run(binding, x)
        assert max_rel_err(got, want) <= 2e-2
    assert rt.last_error() == 0
