"""fp32 mode's tensors in three planes of bf16 parts: every call that writes or reads one, at the edges of
its tiles, against the CPU oracle -- call by call, recorded, and replayed."""
import numpy as np
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


def block(N, C, H, W, K, pool):
    g = graphs.Graph((N, C, H, W), seed=N + C + K)
    v = g.relu(g.conv(0, *g.he_conv(K, C, 7, 7), pads=(3, 3), strides=(2, 2)))
    if pool == "max":
        v = g.maxpool(v, (3, 3), (1, 1), (2, 2))
    elif pool == "avg":
        v = g.avgpool(v, (2, 2), (0, 0), (2, 2))
    y = g.relu(g.conv(v, *g.he_conv(K, K, 3, 3), pads=(1, 1)))
    y = g.conv(y, *g.he_conv(K, K, 1, 1))
    v = g.relu(g.add(y, v))
    v = g.clip(g.conv(v, *g.he_conv(K + 16, K, 1, 1), strides=(2, 2)), 0.0, 6.0)
    return g, v


# (N, C, H, W, K): few-channel and plain inputs; channel counts with and without a plane form, above and
# below a tile; ragged rows; a reduction that is shared by several CTAs
SHAPES = [(1, 3, 65, 47, 64), (2, 3, 40, 72, 48), (3, 16, 33, 33, 144), (1, 5, 32, 64, 40), (5, 3, 64, 64, 256)]


@pytest.mark.parametrize("pool", ["max", "avg", "none"])
@pytest.mark.parametrize("shape", SHAPES)
def test_block(binding, shape, pool):
    g, v = block(*shape, pool)
    g.mark_output(g.linear(g.flatten(g.gap(v)), shape[4] + 16, 24))
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(rt.MATH_FP32)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    for _ in range(4):
        (got,) = p.run(binding, x)
        assert max_rel_err(got, want) <= 5e-5
    assert rt.last_error() == 0


def test_plain_reader(binding):
    """A tensor that a softmax reads leaves the planes."""
    g, v = block(2, 3, 48, 48, 64, "max")
    g.mark_output(g.softmax(v, axis=1))
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(rt.MATH_FP32)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    for _ in range(4):
        (got,) = p.run(binding, x)
        assert np.abs(got - want).max() <= 5e-5
    assert rt.last_error() == 0
