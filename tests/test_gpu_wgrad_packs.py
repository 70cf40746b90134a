"""The tensor-core weight gradient of few input channels, whose MMAs hold several taps
along a kernel's columns, against the oracle in float64: one to eight 8-channel chunks
(rounded up to a power of two), packs that are full, that end early and of one tap,
stride phases with different numbers of taps, and kernels larger than the input.
BF16 <= 1e-2, split BF16 <= 1e-5 of max|oracle|."""

import numpy as np
import pytest

from gpu_util import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu
TOL = {"bf16": 1e-2, "bf16x3": 1e-5}

# input, kernel, stride
CASES = [
    ((2, 21, 30, 8), (5, 18, 8, 16), (1, 1)),        # one chunk: packs of sixteen
    ((2, 18, 25, 16), (2, 9, 16, 24), (1, 1)),       # two chunks: eight and one
    ((3, 30, 13, 24), (7, 6, 24, 40), (1, 1)),       # three chunks of four: four and two
    ((2, 33, 28, 40), (3, 3, 40, 136), (1, 1)),      # five chunks of eight: two and one
    ((1, 40, 41, 64), (5, 5, 64, 64), (1, 1)),
    ((2, 37, 29, 32), (5, 7, 32, 48), (2, 3)),       # phases of three, two and one tap
    ((2, 26, 26, 16), (4, 4, 16, 8), (3, 2)),
    ((5, 4, 3, 32), (6, 5, 32, 16), (1, 1)),         # kernel larger than the input
    ((2, 9, 10, 11, 32), (3, 3, 3, 32, 64), (1, 1, 1)),
    ((1, 11, 12, 13, 8), (2, 5, 3, 8, 24), (2, 2, 1)),
]


@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
@pytest.mark.parametrize("x,w,stride", CASES)
def test_packed_taps(gpu_lib, oracle_nn, prec, x, w, stride):
    from owl_gb300.dense import NN, GpuBackend

    rng = np.random.default_rng(sum(x) * 11 + sum(w))
    o, n, s = oracle_nn, NN(GpuBackend(prec)), list(stride)
    X = rng.uniform(-1, 1, x).astype(np.float32)
    W = rng.standard_normal(w).astype(np.float32)
    X8, W8 = X.astype(np.float64), W.astype(np.float64)
    fwd, grad = ((o.conv3d, o.conv3d_backward_kernel) if len(s) == 3
                 else (o.conv2d, o.conv2d_backward_kernel))
    dy = rng.standard_normal(fwd(X8, W8, s).shape).astype(np.float32)
    ref = grad(X8, W8, s, dy.astype(np.float64))
    f = n.conv3d_backward_kernel if len(s) == 3 else n.conv2d_backward_kernel
    got = from_dev(f(to_dev(X), to_dev(W), s, to_dev(dy)))
    assert gpu_lib.owlgpu_last_conv_path() == 1
    assert rel(got, ref) <= TOL[prec]
    assert gpu_lib.owlgpu_device_status() == 0
