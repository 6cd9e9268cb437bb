"""3x3 convolutions on 64 -> 64 channels whose tiles are column strips of the image (bf16), at ragged widths and
heights, against the CPU oracle."""
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shortcut", [False, True])
@pytest.mark.parametrize("N,H,W", [(40, 15, 17), (30, 33, 131), (24, 64, 65), (8, 61, 255), (100, 14, 14), (3, 112, 224)])
def test_conv(binding, N, H, W, shortcut):
    """conv + bias (+ input) + ReLU; batches large enough for the persistent kernel."""
    g = graphs.Graph((N, 64, H, W), seed=N + H + W)
    y = g.conv(0, *g.he_conv(64, 64, 3, 3), pads=(1, 1))
    g.mark_output(g.relu(g.add(y, g.relu(0)) if shortcut else y))
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(rt.MATH_BF16)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    n0 = rt.form_counters()["column_strips"]
    for _ in range(3):
        (got,) = p.run(binding, x)
        assert max_rel_err(got, want) <= 2e-2
    assert rt.form_counters()["column_strips"] == n0 + 3
    assert rt.last_error() == 0
