"""The float32 vector convolution's three tiles, with windows of 1 to 72 taps: in the
128 x 32 tile a pixel's taps inside the input are a mask that is rebuilt every 32 taps.
Sizes are chosen for the tile named with them on 152 SMs, rows and columns ragged.  A
result has the bits of the scalar kernel's, which operands off a 16-byte boundary take
(k ascending, one fused multiply-add each), and is within 1e-4 of max|oracle|."""

import numpy as np
import pytest

from gpu_util import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu

# input, kernel, stride, rate
CASES = [
    ((1, 84, 71, 16), (7, 5, 16, 160), (1, 1), (1, 1)),      # 128 x 32: 35 taps
    ((2, 61, 34, 16), (9, 8, 16, 256), (1, 1), (1, 1)),      # 128 x 32: 72 taps, three masks
    ((1, 123, 95, 32), (6, 6, 32, 164), (2, 1), (1, 1)),     # 128 x 32: 36 taps, stride
    ((3, 45, 46, 16), (11, 3, 16, 160), (1, 1), (2, 3)),     # 128 x 32: 33 taps, rate
    ((1, 18, 17, 20, 16), (4, 3, 4, 16, 160), (1, 1, 1), None),  # 128 x 32: 48 taps
    ((3, 70, 59, 16), (3, 3, 16, 256), (1, 1), (1, 1)),      # 128 x 64
    ((2, 91, 69, 32), (1, 2, 32, 244), (1, 1), (1, 1)),      # 128 x 64, ragged columns
    ((2, 23, 29, 48), (8, 5, 48, 68), (1, 1), (1, 1)),       # 64 x 32: 40 taps
]


def _off(a):
    """The same values 4 bytes past a 16-byte boundary."""
    import torch

    flat = torch.empty(a.size + 1, device="cuda")[1:]
    flat.copy_(torch.from_numpy(np.ascontiguousarray(a)).reshape(-1))
    return flat.reshape(a.shape)


@pytest.mark.parametrize("x,w,stride,rate", CASES)
def test_tiles_and_masks(gpu_lib, oracle_nn, x, w, stride, rate):
    from owl_gb300.dense import NN, GpuBackend

    G, s = NN(GpuBackend("fp32")), list(stride)
    if rate is None:
        fwd, grad = (lambda n, a, b: n.conv3d(a, b, s),
                     lambda a, b, d: G.conv3d_backward_kernel(a, b, s, d))
    else:
        r = list(rate)
        fwd, grad = (lambda n, a, b: n.dilated_conv2d(a, b, s, r),
                     lambda a, b, d: G.dilated_conv2d_backward_kernel(a, b, s, r, d))
    rng = np.random.default_rng(sum(x) + sum(w))
    X = rng.uniform(-1, 1, x).astype(np.float32)
    W = rng.uniform(-1, 1, w).astype(np.float32)
    y = from_dev(fwd(G, to_dev(X), to_dev(W)))
    np.testing.assert_array_equal(from_dev(fwd(G, _off(X), to_dev(W))), y)
    assert rel(y, fwd(oracle_nn, X, W)) <= 1e-4
    D = rng.uniform(-1, 1, y.shape).astype(np.float32)
    dw = from_dev(grad(to_dev(X), to_dev(W), to_dev(D)))
    np.testing.assert_array_equal(from_dev(grad(_off(X), to_dev(W), to_dev(D))), dw)
