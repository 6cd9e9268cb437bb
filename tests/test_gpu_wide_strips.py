"""3x3 layers with up to 128 output channels as column strips (weights on the M side): image sizes that no strip divides,
channel counts with remainders, several 64-channel blocks, one tile and many waves, clamps, and 2x2 max pools taken along.
Inputs and filters are bf16 numbers, so that only the result is rounded: a bf16 has eight bits, half a step of the
last is at most 2^-8 of the value."""
import numpy as np
import pytest

from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu


def _bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("N,C,H,W,K,act,pool", [
    (24, 128, 28, 28, 128, "relu", False),
    (61, 128, 26, 26, 128, "relu", False),
    (40, 64, 57, 45, 128, "clip", False),     # one block of channels; a last strip and a last row band that reach out
    (37, 192, 31, 17, 72, None, False),       # three blocks; channels with a remainder
    (33, 128, 40, 33, 64, "relu", False),     # one slab of channels
    (8, 64, 112, 112, 128, "relu", False),
    (150, 128, 15, 9, 104, "relu", False),
    (8, 128, 112, 112, 128, "relu", True),
    (40, 128, 57, 31, 128, "relu", True),     # odd heights and widths: the pool leaves the last ones out
    (8, 64, 112, 112, 96, None, True),
])
def test_wide(binding, N, C, H, W, K, act, pool):
    g = graphs.Graph((N, C, H, W), seed=N + C + H)
    w, b = g.he_conv(K, C, 3, 3)
    v = g.conv(0, _bf16(w), b, pads=(1, 1))
    v = g.relu(v) if act == "relu" else g.clip(v, -0.75, 1.25) if act == "clip" else v
    if pool:
        v = g.maxpool(v, (2, 2), (0, 0), (2, 2))
    g.mark_output(v)
    x = _bf16(graphs.make_input(g, 1))
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(rt.MATH_BF16)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    before = rt.form_counters()
    got = [p.run(binding, x)[0] for _ in range(4)]
    after = rt.form_counters()
    assert after["column_strips"] - before["column_strips"] >= 3
    assert (after["pooled"] - before["pooled"] >= 3) == pool
    for y in got[2:]:   # (the first is made call by call: bias and clamp round again)
        assert max_rel_err(y, want) <= 2.0 ** -8 * 1.02   # (and what sums in another order differ by)
        assert np.array_equal(y, got[2])
    assert rt.last_error() == 0


@pytest.mark.parametrize("N,C,H,W,K", [(600, 128, 7, 6, 128), (700, 64, 4, 4, 128), (900, 192, 9, 8, 72), (2000, 128, 8, 8, 64)])
def test_small_images_share_tiles(binding, N, C, H, W, K):
    """Images much smaller than a tile go to the form whose tiles hold several."""
    g = graphs.Graph((N, C, H, W), seed=N + C + H)
    w, b = g.he_conv(K, C, 3, 3)
    g.mark_output(g.relu(g.conv(0, _bf16(w), b, pads=(1, 1))))
    x = _bf16(graphs.make_input(g, 1))
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(rt.MATH_BF16)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    before = rt.form_counters()["column_strips"]
    got = [p.run(binding, x)[0] for _ in range(3)]
    assert rt.form_counters()["column_strips"] == before
    for y in got:
        assert max_rel_err(y, want) <= 2.0 ** -8 * 1.02
    assert rt.last_error() == 0
