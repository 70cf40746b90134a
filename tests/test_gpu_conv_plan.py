"""The tensor-core convolution's tile choice over batch sizes, against the oracle
in float64: batches whose tiles leave SMs idle, fill them and go round several
times; outputs of 1 to 70 rows (tiles of 2 to 32), one, two and three co tiles,
channels of one block, of several and of ragged ones, and halos that fit only with
a narrow block or a low tile.  The same bits for an entry whatever its batch.
BF16 <= 1e-2, split BF16 <= 1e-5 of max|oracle|."""

import numpy as np
import pytest

from gpu_util import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu
TOL = {"bf16": 1e-2, "bf16x3": 1e-5}

# rows x columns, channels in and out, kernel, stride, rate, largest batch
CASES = [
    ((1, 9), 16, 24, (1, 3), 1, 1, 300),
    ((7, 7), 264, 264, (3, 3), 1, 1, 40),
    ((14, 13), 136, 384, (1, 1), 2, 1, 90),
    ((33, 10), 112, 130, (3, 3), 1, 1, 20),
    ((31, 17), 104, 16, (2, 2), 2, 1, 50),
    ((70, 9), 80, 40, (3, 3), 1, 1, 30),
    ((64, 24), 32, 16, (3, 3), 2, 1, 20),
    ((24, 24), 64, 24, (3, 3), 1, 7, 12),
]


@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
@pytest.mark.parametrize("hw,ci,co,k,s,r,most", CASES)
def test_tile_choice(gpu_lib, oracle_nn, prec, hw, ci, co, k, s, r, most):
    from owl_gb300.dense import NN, GpuBackend

    rng = np.random.default_rng(ci * 3 + co)
    N, st, rt = NN(GpuBackend(prec)), [s, s], [r, r]
    X = rng.uniform(-1, 1, (most,) + hw + (ci,)).astype(np.float32)
    W = (rng.standard_normal(k + (ci, co)) * np.sqrt(2 / (k[0] * k[1] * ci))).astype(np.float32)
    X8, W8 = X[:2].astype(np.float64), W.astype(np.float64)
    y = oracle_nn.dilated_conv2d(X8, W8, st, rt)
    dy = rng.standard_normal((most,) + y.shape[1:]).astype(np.float32)
    dx = oracle_nn.dilated_conv2d_backward_input(X8, W8, st, rt, dy[:2].astype(np.float64))
    Xd, Wd, Dd = to_dev(X), to_dev(W), to_dev(dy)
    first = None
    for n in (most, most // 3, 2):
        got = []
        for f in (lambda: N.dilated_conv2d(Xd[:n], Wd, st, rt),
                  lambda: N.dilated_conv2d_backward_input(Xd[:n], Wd, st, rt, Dd[:n])):
            got.append(from_dev(f())[:2])
            assert gpu_lib.owlgpu_last_conv_path() == 1
        if first is None:
            first = got
            assert rel(got[0], y) <= TOL[prec] and rel(got[1], dx) <= TOL[prec]
        np.testing.assert_array_equal(got[0], first[0])
        np.testing.assert_array_equal(got[1], first[1])
    assert gpu_lib.owlgpu_device_status() == 0
