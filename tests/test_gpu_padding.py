"""The two passes that give an image the form its convolution reads, at ragged sizes, against the CPU oracle:
few channels interleaved and bordered, and channels appended up to a multiple of sixteen."""
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


# rows in all: not a multiple of a block's eight, images that end inside a block and inside four rows of it
@pytest.mark.parametrize("mode", [rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("N,C,H,W,K,R,stride", [(1, 3, 131, 97, 32, 3, 2), (7, 3, 45, 61, 64, 7, 2), (21, 1, 11, 200, 64, 3, 1),
                                                (300, 3, 7, 9, 64, 3, 1), (5, 6, 33, 40, 64, 3, 1), (2, 12, 30, 71, 32, 5, 1),
                                                (2, 24, 29, 31, 64, 1, 1), (9, 40, 17, 13, 96, 3, 1), (33, 72, 57, 56, 32, 1, 1)])
def test_padded_input(binding, N, C, H, W, K, R, stride, mode):
    g = graphs.Graph((N, C, H, W), seed=N + C + H)
    y = g.conv(0, *g.he_conv(K, C, R, R), pads=(R // 2, R // 2), strides=(stride, stride))
    g.mark_output(g.relu(y))
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    for _ in range(3):
        (got,) = p.run(binding, x)
        assert max_rel_err(got, want) <= 2e-2
    assert rt.last_error() == 0
