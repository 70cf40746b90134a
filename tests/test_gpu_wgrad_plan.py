"""The tensor-core weight gradient's plan and staging tables at their edges, against
the oracle in float64: tap groups of one to sixteen taps, output blocks of 16 to 256
channels, tiles of one and of several staging rounds, heights of 2 to 16 rows that
leave rows over, kernels larger than the input, several tiles along every axis, and
one pixel range or many.  The same bits on a second call.  BF16 <= 1e-2, split BF16
<= 1e-5 of max|oracle|."""

import numpy as np
import pytest

from gpu_util import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu
TOL = {"bf16": 1e-2, "bf16x3": 1e-5}

# input, kernel, stride, rate
CASES = [
    ((9, 1, 8, 8), (1, 1, 8, 16), (1, 1), (1, 1)),         # one tap, one row
    ((2, 5, 6, 16), (9, 7, 16, 24), (1, 1), (1, 1)),       # kernel larger than the input
    ((3, 29, 31, 136), (3, 3, 136, 40), (1, 1), (1, 1)),   # two input blocks
    ((2, 19, 23, 16), (4, 4, 16, 264), (1, 1), (1, 1)),    # two output blocks, 16 taps
    ((1, 34, 50, 128), (3, 3, 128, 128), (1, 1), (6, 5)),  # several rounds a tile
    ((2, 47, 18, 64), (5, 1, 64, 72), (3, 1), (1, 1)),
    ((40, 15, 9, 24), (3, 3, 24, 56), (2, 2), (1, 1)),     # many pixel ranges
    ((1, 70, 9, 8), (2, 17, 8, 8), (1, 2), (1, 1)),        # many taps in a row
    ((2, 6, 17, 19, 32), (3, 3, 3, 32, 64), (1, 1, 1), (1, 1, 1)),
    ((3, 7, 9, 8, 16), (2, 3, 4, 16, 8), (2, 1, 3), (1, 1, 1)),
]


@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
@pytest.mark.parametrize("x,w,stride,rate", CASES)
def test_weight_gradient(gpu_lib, oracle_nn, prec, x, w, stride, rate):
    from owl_gb300.dense import NN, GpuBackend

    rng = np.random.default_rng(sum(x) * 5 + sum(w))
    s, r = list(stride), list(rate)
    three = len(s) == 3
    o, n = oracle_nn, NN(GpuBackend(prec))

    def out(lib, X, W):
        return lib.conv3d(X, W, s) if three else lib.dilated_conv2d(X, W, s, r)

    def grad(lib, X, W, D):
        if three:
            return lib.conv3d_backward_kernel(X, W, s, D)
        return lib.dilated_conv2d_backward_kernel(X, W, s, r, D)

    X = rng.uniform(-1, 1, x).astype(np.float32)
    W = rng.standard_normal(w).astype(np.float32)
    X8, W8 = X.astype(np.float64), W.astype(np.float64)
    dy = rng.standard_normal(out(o, X8, W8).shape).astype(np.float32)
    ref = grad(o, X8, W8, dy.astype(np.float64))
    Xd, Wd, Dd = to_dev(X), to_dev(W), to_dev(dy)
    got = from_dev(grad(n, Xd, Wd, Dd))
    assert gpu_lib.owlgpu_last_conv_path() == 1
    assert rel(got, ref) <= TOL[prec]
    np.testing.assert_array_equal(from_dev(grad(n, Xd, Wd, Dd)), got)
    assert gpu_lib.owlgpu_device_status() == 0
