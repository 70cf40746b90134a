"""The tensor-core GEMM's tile widths and splits: products whose plans take tiles
from 16 to 256 columns, ragged last tiles, one and many splits, against float64
(BF16 <= 1e-2, split BF16 <= 1e-5 of the products' magnitude), the same bits on
every run."""

import numpy as np
import pytest

from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu

SIZES = [(3136, 1024, 256), (256, 3136, 1024), (256, 1024, 3136), (129, 200, 700), (1, 16, 64),
         (4096, 24, 100), (640, 488, 65), (128, 8, 8192), (257, 257, 257), (2000, 2000, 128)]


@pytest.mark.parametrize("prec,tol", [("bf16", 1e-2), ("bf16x3", 1e-5)])
@pytest.mark.parametrize("m,n,k", SIZES)
def test_gemm_plans(gpu_lib, prec, tol, m, n, k):
    from owl_gb300.dense import NN, GpuBackend
    from owl_gb300.layers import ACT_RELU, Layers

    L = Layers(NN(GpuBackend(prec)))
    rng = np.random.default_rng(m * 3 + n * 5 + k)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    bias = rng.uniform(-1, 1, n).astype(np.float32)
    exact = a.astype(np.float64) @ b.astype(np.float64)
    scale = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    for ta, tb in ((False, False), (False, True), (True, False)):
        A = to_dev(np.ascontiguousarray(a.T) if ta else a)
        B = to_dev(np.ascontiguousarray(b.T) if tb else b)
        c = from_dev(L.dot(A, B, trans_a=ta, trans_b=tb))
        assert np.max(np.abs(c - exact) / scale) <= tol, (ta, tb)
        np.testing.assert_array_equal(from_dev(L.dot(A, B, trans_a=ta, trans_b=tb)), c)
        z = from_dev(L.dot(A, B, trans_a=ta, trans_b=tb, bias=to_dev(bias), act=ACT_RELU))
        np.testing.assert_array_equal(z, np.maximum(c + bias, 0))
