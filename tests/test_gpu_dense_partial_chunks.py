"""Dense products on the tensor cores whose row-contiguous operands end inside an
8-row chunk (M or N a multiple of 4 but not of 8, rows 16-byte aligned), with
whole 64-deep k blocks: the last rows and columns take part like the others."""

import numpy as np
import pytest

from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("bf16", 1e-2), ("bf16x3", 1e-5)])
@pytest.mark.parametrize("m,n,k", [(164, 100, 800), (100, 36, 512), (12, 260, 192), (68, 4, 64)])
def test_partial_row_chunks(gpu_lib, prec, tol, m, n, k):
    from owl_gb300.dense import NN, GpuBackend
    from owl_gb300.layers import Layers

    L = Layers(NN(GpuBackend(prec)))
    rng = np.random.default_rng(m + n + k)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    exact = a.astype(np.float64) @ b.astype(np.float64)
    scale = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    for ta, tb in ((False, False), (False, True), (True, False)):
        A = to_dev(np.ascontiguousarray(a.T) if ta else a)
        B = to_dev(np.ascontiguousarray(b.T) if tb else b)
        c = from_dev(L.dot(A, B, trans_a=ta, trans_b=tb))
        assert np.max(np.abs(c - exact) / scale) <= tol, (ta, tb)
