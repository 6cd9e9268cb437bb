"""Large batches from host memory, which are computed in pieces while they arrive: every pass with another
batch, and with a constant that changes, against the same model computed from device memory."""
import numpy as np
import pytest
import torch

from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt

pytestmark = pytest.mark.gpu

PASSES = 9


def net(N, size):
    g = graphs.Graph((N, 3, size, size), seed=N)
    v = g.relu(g.conv(0, *g.he_conv(64, 3, 7, 7), pads=(3, 3), strides=(2, 2)))
    v = g.maxpool(v, (3, 3), (1, 1), (2, 2))
    y = g.relu(g.conv(v, *g.he_conv(64, 64, 3, 3), pads=(1, 1)))
    v = g.relu(g.add(g.conv(y, *g.he_conv(64, 64, 1, 1)), v))
    g.mark_output(g.linear(g.flatten(g.gap(v)), 64, 40))
    return g


@pytest.mark.parametrize("fuse", [replay.FUSE_REFERENCE, replay.FUSE_NONE])
@pytest.mark.parametrize("math", [rt.MATH_BF16, rt.MATH_F16, rt.MATH_FP32])
@pytest.mark.parametrize("N,size", [(128, 112), (151, 121), (127, 112)])
def test_batches(binding, N, size, math, fuse):
    g = net(N, size)
    rt.set_math_mode(math)
    p = g.to_program()
    p.lower(fuse=fuse)
    rng = np.random.default_rng(N)
    xs = [rng.standard_normal(g.input_shape, dtype=np.float32) for _ in range(2)]
    head = max(g.consts, key=lambda k: g.consts[k].size == 64 * 40)
    for i in range(PASSES):
        if i == PASSES - 2:   # the classifier's weights, in place
            g.consts[head] *= 0.5
        x = torch.from_numpy(xs[i % 2] * (1 + i)).pin_memory()
        (got,) = p.run(binding, x.numpy())
        dev = x.cuda()
        want = torch.empty(g.shapes[g.outputs[0]], device="cuda")
        torch.cuda.synchronize()
        p.run_raw(binding, dev.data_ptr(), 3, [want.data_ptr()], 3)
        rt.synchronize()
        want = want.cpu().numpy()
        assert np.abs(got - want).max() <= {rt.MATH_FP32: 2e-5, rt.MATH_F16: 1e-3}.get(math, 8e-3) * np.abs(want).max()
    assert rt.last_error() == 0
