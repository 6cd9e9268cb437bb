"""The split-reduction convolution / GEMM kernel (few output tiles, a cluster of CTAs per tile) at the
edges of its tiles and of its splits, against the CPU oracle."""
import numpy as np
import pytest

from calls import Inference, rand
from helpers import max_rel_err, run_graph_oracle
from occamy_b200 import graphs, replay
from occamy_b200 import runtime as rt
from oracle import ref

pytestmark = pytest.mark.gpu

TOL = {rt.MATH_FP32: 1e-4, rt.MATH_BF16: 2e-2, rt.MATH_F16: 2e-2}

# (N, C, H, W, K, R, stride): reductions of 1 to 72 k-steps in 1 to 8 shares, equal or not; tiles of 1
# to 128 pixels, several images per tile, channel counts that leave a partial last tile
SHAPES = [
    (1, 16, 1, 1, 8, 1, 1),
    (1, 64, 7, 7, 40, 1, 1),
    (1, 512, 7, 7, 512, 3, 1),
    (3, 512, 7, 7, 200, 3, 1),
    (2, 448, 5, 9, 72, 3, 2),
    (1, 2048, 7, 7, 136, 1, 1),
    (2, 272, 13, 11, 96, 3, 1),
    (4, 96, 12, 12, 264, 3, 1),
    (1, 1024, 14, 14, 256, 1, 2),
]


@pytest.mark.parametrize("mode", sorted(TOL))
@pytest.mark.parametrize("shape", SHAPES)
def test_conv_with_residual(binding, shape, mode):
    """conv + bias + shortcut + ReLU, as separate calls and (third pass) as one kernel."""
    N, C, H, W, K, R, st = shape
    g = graphs.Graph((N, C, H, W), seed=sum(shape))
    ws, bs = g.he_conv(K, C, 1, 1)
    short = g.conv(0, ws, bs, strides=(st, st))
    w, b = g.he_conv(K, C, R, R)
    y = g.conv(0, w, b, pads=(R // 2, R // 2), strides=(st, st))
    g.mark_output(g.relu(g.add(y, short)))
    x = graphs.make_input(g, 1)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    n0 = rt.form_counters()["split_reduction"]
    for _ in range(3):
        (got,) = p.run(binding, x)
        assert max_rel_err(got, want) <= TOL[mode]
    if mode != rt.MATH_FP32 or N * H * W * C * K * R * R >= 1e6 * st * st:   # (smaller ones stay on the CUDA cores)
        assert rt.form_counters()["split_reduction"] >= n0 + 3
    assert rt.last_error() == 0


@pytest.mark.parametrize("mode", sorted(TOL))
@pytest.mark.parametrize("M,K,N", [(1, 2048, 1000), (5, 4096, 4096), (33, 1280, 10), (128, 512, 1000), (130, 4096, 36)])
def test_gemm(binding, M, K, N, mode):
    g = graphs.Graph((M, K), seed=M + N)
    g.mark_output(g.linear(0, K, N))
    x = graphs.make_input(g, 2)
    (want,) = run_graph_oracle(g, x)
    rt.set_math_mode(mode)
    p = g.to_program()
    p.lower(fuse=replay.FUSE_REFERENCE)
    n0 = rt.form_counters()["split_reduction"]
    for _ in range(2):
        (got,) = p.run(binding, x)
        assert max_rel_err(got, want) <= TOL[mode]
    if mode != rt.MATH_FP32 or M * K * N >= 1e6:
        assert rt.form_counters()["split_reduction"] == n0 + 2
    assert rt.last_error() == 0


@pytest.mark.parametrize("mode", [rt.MATH_FP32, rt.MATH_BF16, rt.MATH_F16])
@pytest.mark.parametrize("act", [1, 5])
def test_nan_stays(native_libs, mode, act):
    """ReLU and no activation keep NaN, in the kernels for few tiles as well."""
    rt.set_math_mode(mode)
    w, b = rand(1, 64, 64, 3, 3, scale=0.1), rand(2, 64)
    fc = rand(3, 48, 64, scale=0.1)
    x = rand(4, 2, 64, 14, 14)
    x[0, 3, 5, 6] = np.nan
    m = rand(5, 4, 64)
    m[1, 7] = np.nan
    want, want2 = ref.conv2d(x, w, b, (1, 1), act=act), ref.matmul2d(m, fc, transB=1)
    if act == 1:
        want2 = np.where(np.isnan(want2), want2, np.maximum(want2, 0))
    for i in range(4):
        with Inference() as f:
            y, o = f.conv(f.put(x), x.shape, f.put(w), w.shape, f.put(b), (1, 1), act=act)
            got = f.get(y, o)
            y, o = f.matmul(f.put(m), m.shape, f.put(fc), fc.shape)
            if act == 1:
                y2 = f.place(int(np.prod(o)) * 4)
                rt.lib().DNNActiveFunc(f.h, y, rt.dims(o + (1, 1)), 1, y2)
                y = y2
            got2 = f.get(y, o)
        for g, t in ((got, want), (got2, want2)):
            assert np.array_equal(np.isnan(g), np.isnan(t)), i
            ok = ~np.isnan(t)
            assert max_rel_err(g[ok], t[ok]) <= 2e-2
    assert rt.last_error() == 0
