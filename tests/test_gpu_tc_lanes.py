"""The tensor-core kernels' staging in whole 32-byte chunks at its edges, against
the oracle in float64: channel counts whose chunks are and are not a power of two
(one to sixteen a block, ragged last blocks), rows of one to many rounds, stride
phases of which only some are read, 3-D halos of more rows than producer warps;
and operands that are not 32-byte aligned, which take the element-wise staging to
the same bits.  BF16 <= 1e-2, split BF16 <= 1e-5 of max|oracle|."""

import numpy as np
import pytest

from gpu_util import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu
TOL = {"bf16": 1e-2, "bf16x3": 1e-5}

# input, kernel, stride, rate
CASES = [
    ((2, 9, 11, 8), (3, 3, 8, 8), (1, 1), (1, 1)),        # one chunk
    ((2, 13, 17, 24), (3, 3, 24, 40), (1, 1), (1, 1)),    # three and five chunks
    ((1, 16, 16, 72), (3, 3, 72, 136), (1, 1), (1, 1)),   # nine and seventeen chunks
    ((1, 15, 20, 200), (1, 1, 200, 264), (1, 1), (1, 1)),
    ((2, 20, 19, 32), (1, 1, 32, 64), (2, 2), (1, 1)),    # a quarter of the rows is read
    ((2, 21, 23, 40), (2, 1, 40, 16), (3, 2), (1, 1)),    # two of three phases, one of two
    ((1, 30, 29, 16), (5, 5, 16, 24), (2, 2), (1, 1)),
    ((1, 24, 40, 16), (3, 3, 16, 32), (1, 1), (4, 9)),    # wide rows: several rounds
    ((1, 40, 9, 128), (7, 7, 128, 16), (1, 1), (1, 1)),
    ((3, 5, 6, 7, 24), (3, 3, 3, 24, 40), (1, 1, 1), (1, 1, 1)),
    ((1, 12, 11, 10, 32), (3, 3, 3, 32, 16), (2, 2, 2), (1, 1, 1)),
    ((2, 4, 1, 33, 48), (1, 1, 5, 48, 24), (1, 1, 1), (1, 1, 1)),
]


def _calls(N, nd, stride, rate):
    if nd == 2:
        s, r = list(stride), list(rate)
        return (lambda x, w: N.dilated_conv2d(x, w, s, r),
                lambda x, w, d: N.dilated_conv2d_backward_input(x, w, s, r, d),
                lambda x, w, d: N.dilated_conv2d_backward_kernel(x, w, s, r, d))
    s = list(stride)
    return (lambda x, w: N.conv3d(x, w, s),
            lambda x, w, d: N.conv3d_backward_input(x, w, s, d),
            lambda x, w, d: N.conv3d_backward_kernel(x, w, s, d))


def _unaligned(a):
    """The same values 4 bytes past a 32-byte boundary."""
    import torch

    flat = torch.empty(a.size + 1, device="cuda")[1:]
    flat.copy_(torch.from_numpy(np.ascontiguousarray(a)).reshape(-1))
    return flat.reshape(a.shape)


@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
@pytest.mark.parametrize("x,w,stride,rate", CASES)
def test_lane_staging(gpu_lib, oracle_nn, prec, x, w, stride, rate):
    from owl_gb300.dense import NN, GpuBackend

    rng = np.random.default_rng(sum(x) * 7 + sum(w))
    X = rng.uniform(-1, 1, x).astype(np.float32)
    W = (rng.standard_normal(w) * np.sqrt(2 / np.prod(w[:-1]))).astype(np.float32)
    nd = len(stride)
    of, oi, ok = _calls(oracle_nn, nd, stride, rate)
    gf, gi, gk = _calls(NN(GpuBackend(prec)), nd, stride, rate)
    X8, W8 = X.astype(np.float64), W.astype(np.float64)
    y = of(X8, W8)
    dy = rng.standard_normal(y.shape).astype(np.float32)
    ref = (y, oi(X8, W8, dy.astype(np.float64)), ok(X8, W8, dy.astype(np.float64)))
    Xd, Wd, Dd = to_dev(X), to_dev(W), to_dev(dy)
    got = []
    for f, r in ((lambda: gf(Xd, Wd), ref[0]), (lambda: gi(Xd, Wd, Dd), ref[1]),
                 (lambda: gk(Xd, Wd, Dd), ref[2])):
        a = from_dev(f())
        assert gpu_lib.owlgpu_last_conv_path() == 1
        assert rel(a, r) <= TOL[prec]
        got.append(a)
    Xu, Du = _unaligned(X), _unaligned(dy)
    np.testing.assert_array_equal(from_dev(gf(Xu, Wd)), got[0])
    np.testing.assert_array_equal(from_dev(gi(Xu, Wd, Du)), got[1])
    np.testing.assert_array_equal(from_dev(gk(Xu, Wd, Du)), got[2])
    assert gpu_lib.owlgpu_device_status() == 0
