"""The CUDA-core convolutions and dense products at the edges of their tiles and
split sums, against the oracle: windows of more than 32 taps (the tap masks are
rebuilt), reductions longer than the scalar kernel's tap table, one-channel
backward_kernels, the float64 tiles, x w^T products, fused bias and ReLU, and sums
of few and many partials.  float32 <= 1e-4, float64 <= 1e-11 of max|oracle|."""

import numpy as np
import pytest

from gpu_util import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu
TOL = {np.float32: 1e-4, np.float64: 1e-11}

# input, kernel, stride, rate
CONVS = [
    ((2, 9, 11, 16), (7, 5, 16, 24), (1, 1), (1, 1)),     # 35 taps, vector path
    ((1, 13, 12, 32), (8, 8, 32, 68), (1, 2), (1, 1)),    # 64 taps: three mask words
    ((2, 17, 19, 7), (5, 5, 7, 9), (1, 1), (1, 1)),       # scalar, 175 k
    ((1, 12, 10, 30), (5, 5, 30, 33), (2, 1), (1, 1)),    # scalar, 750 k: two tables
    ((3, 28, 27, 1), (5, 5, 1, 32), (1, 1), (1, 1)),      # one channel: 25 kernel rows
    ((2, 20, 21, 1), (6, 6, 1, 5), (1, 1), (1, 1)),       # 36 kernel rows
    ((2, 14, 15, 3), (3, 3, 3, 40), (2, 2), (1, 1)),
    ((2, 31, 33, 48), (3, 3, 48, 36), (1, 1), (2, 2)),
    ((1, 70, 64, 32), (1, 1, 32, 160), (1, 1), (1, 1)),
]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("x,w,stride,rate", CONVS)
def test_conv_tiles(oracle_nn, gpu_lib, dt, x, w, stride, rate):
    from owl_gb300.dense import NN, GpuBackend

    G, O = NN(GpuBackend("fp32")), oracle_nn
    rng = np.random.default_rng(sum(x) + sum(w))
    X = rng.uniform(-1, 1, x).astype(dt)
    W = rng.uniform(-1, 1, w).astype(dt)
    s, r = list(stride), list(rate)
    y = O.dilated_conv2d(X, W, s, r)
    dy = rng.uniform(-1, 1, y.shape).astype(dt)
    Xd, Wd, dyd = to_dev(X), to_dev(W), to_dev(dy)
    got = {
        "fwd": (from_dev(G.dilated_conv2d(Xd, Wd, s, r)), y),
        "bwd_input": (from_dev(G.dilated_conv2d_backward_input(Xd, Wd, s, r, dyd)),
                      O.dilated_conv2d_backward_input(X, W, s, r, dy)),
        "bwd_kernel": (from_dev(G.dilated_conv2d_backward_kernel(Xd, Wd, s, r, dyd)),
                       O.dilated_conv2d_backward_kernel(X, W, s, r, dy)),
    }
    for name, (a, b) in got.items():
        assert rel(a, b) <= TOL[dt], name


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("m,n,k", [(256, 1024, 3136), (33, 36, 528), (130, 100, 1040), (7, 5, 9),
                                   (64, 260, 16), (1, 4, 4096), (300, 31, 64)])
def test_dense_tiles(gpu_lib, dt, m, n, k):
    from owl_gb300.dense import NN, GpuBackend
    from owl_gb300.layers import ACT_RELU, Layers

    L = Layers(NN(GpuBackend("fp32")))
    rng = np.random.default_rng(m + n + k)
    a = rng.uniform(-1, 1, (m, k)).astype(dt)
    b = rng.uniform(-1, 1, (k, n)).astype(dt)
    bias = rng.uniform(-1, 1, n).astype(dt)
    exact = a.astype(np.float64) @ b.astype(np.float64)
    scale = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    tol = 1e-5 if dt == np.float32 else 1e-12
    for ta, tb in ((False, False), (False, True), (True, False)):
        A = to_dev(np.ascontiguousarray(a.T) if ta else a)
        B = to_dev(np.ascontiguousarray(b.T) if tb else b)
        c = from_dev(L.dot(A, B, trans_a=ta, trans_b=tb))
        assert np.max(np.abs(c - exact) / scale) <= tol, (ta, tb)
        # the bias and ReLU on the finished sums: exactly the two-step result
        z = from_dev(L.dot(A, B, trans_a=ta, trans_b=tb, bias=to_dev(bias), act=ACT_RELU))
        np.testing.assert_array_equal(z, np.maximum(c + bias, 0))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(2, 9, 8, 16, 36), (2, 9, 8, 3, 5)])
def test_conv_bias_act_is_the_two_step_result(gpu_lib, dt, shape):
    from owl_gb300.dense import NN, GpuBackend, SAME
    from owl_gb300.layers import ACT_RELU, Layers

    G = NN(GpuBackend("fp32"))
    b, h, w, ci, co = shape
    rng = np.random.default_rng(ci)
    x = to_dev(rng.uniform(-1, 1, (b, h, w, ci)).astype(dt))
    k = to_dev(rng.uniform(-1, 1, (3, 3, ci, co)).astype(dt))
    bias = rng.uniform(-1, 1, co).astype(dt)
    y = from_dev(G.conv2d(x, k, [1, 1], SAME))
    z = from_dev(Layers(G).conv2d_bias_act(x, k, to_dev(bias), [1, 1], SAME, ACT_RELU))
    np.testing.assert_array_equal(z, np.maximum(y + bias, 0))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("p,c", [(50176, 64), (65, 32), (1, 5), (777, 33), (4096, 2), (129, 68)])
def test_bias_act_backward_edges(gpu_lib, dt, p, c):
    from owl_gb300.dense import NN, GpuBackend
    from owl_gb300.layers import ACT_NONE, ACT_RELU, Layers

    L = Layers(NN(GpuBackend("fp32")))
    rng = np.random.default_rng(p + c)
    y = np.maximum(rng.standard_normal((p, c)), 0).astype(dt)
    dy = rng.standard_normal((p, c)).astype(dt)
    for act, want in ((ACT_RELU, dy * (y > 0)), (ACT_NONE, dy)):
        dz, db = L.bias_act_backward(to_dev(y), to_dev(dy), act)
        np.testing.assert_array_equal(from_dev(dz), want)
        ref = want.astype(np.float64).sum(0)
        scale = np.abs(want.astype(np.float64)).sum(0) + 1e-30
        assert np.max(np.abs(from_dev(db) - ref) / scale) <= (1e-5 if dt == np.float32 else 1e-13)
