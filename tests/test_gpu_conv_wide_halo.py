"""Tensor-core convolutions whose halo fills the shared memory: dilated kernels at
rates where the staging table of its pixels leaves room only for low tiles or for
none, with strides whose phases are all or partly read, against the oracle in
float64.  The passes run on the tensor cores; an entry has the same bits alone and
in its batch, and from operands that are not 32-byte aligned.  BF16 <= 1e-2, split
BF16 <= 1e-5 of max|oracle|."""

import numpy as np
import pytest

from gpu_util import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu
TOL = {"bf16": 1e-2, "bf16x3": 1e-5}

# precision, rows x columns, channels in and out, kernel, stride, rate
CASES = [
    ("bf16", (65, 65), 48, 40, 3, 1, 36),
    ("bf16", (40, 45), 16, 136, 3, 1, 38),
    ("bf16", (50, 41), 24, 24, 5, 1, 18),
    ("bf16", (47, 39), 16, 8, 7, 1, 12),
    ("bf16", (29, 38), 40, 24, 9, 1, 9),
    ("bf16", (33, 30), 64, 72, 3, 1, 25),     # two stages of low tiles, or one of tall
    ("bf16", (32, 13), 16, 136, 7, 2, 7),
    ("bf16", (65, 25), 24, 16, 9, 2, 17),     # forward on the CUDA cores
    ("bf16", (53, 26), 40, 24, 7, 3, 11),
    ("bf16x3", (41, 43), 24, 24, 3, 1, 25),
    ("bf16x3", (31, 37), 64, 40, 3, 1, 17),
    ("bf16x3", (30, 12), 48, 24, 9, 3, 5),
    ("bf16x3", (40, 56), 24, 24, 9, 2, 5),
]


def _unaligned(a):
    """The same values 4 bytes past a 32-byte boundary."""
    import torch

    flat = torch.empty(a.size + 1, device="cuda")[1:]
    flat.copy_(torch.from_numpy(np.ascontiguousarray(a)).reshape(-1))
    return flat.reshape(a.shape)


@pytest.mark.parametrize("prec,hw,ci,co,k,s,r", CASES)
def test_wide_halos(gpu_lib, oracle_nn, prec, hw, ci, co, k, s, r):
    from owl_gb300.dense import NN, GpuBackend

    rng = np.random.default_rng(ci * 5 + co + r)
    N, st, rt = NN(GpuBackend(prec)), [s, s], [r, r]
    X = rng.uniform(-1, 1, (3,) + hw + (ci,)).astype(np.float32)
    W = (rng.standard_normal((k, k, ci, co)) * np.sqrt(2 / (k * k * ci))).astype(np.float32)
    X8, W8 = X[:1].astype(np.float64), W.astype(np.float64)
    y = oracle_nn.dilated_conv2d(X8, W8, st, rt)
    D = rng.standard_normal((3,) + y.shape[1:]).astype(np.float32)
    dx = oracle_nn.dilated_conv2d_backward_input(X8, W8, st, rt, D[:1].astype(np.float64))
    Wd, Xd, Dd = to_dev(W), to_dev(X), to_dev(D)

    def both(x, d):
        out = []
        for f in (lambda: N.dilated_conv2d(x, Wd, st, rt),
                  lambda: N.dilated_conv2d_backward_input(x, Wd, st, rt, d)):
            out.append(from_dev(f()))
            fits = (s, r) != (2, 17) or len(out) == 2
            assert gpu_lib.owlgpu_last_conv_path() == int(fits)
        return out

    got = both(Xd, Dd)
    assert rel(got[0][:1], y) <= TOL[prec] and rel(got[1][:1], dx) <= TOL[prec]
    for a, b in zip(got, both(Xd[:1], Dd[:1])):
        np.testing.assert_array_equal(b, a[:1])
    for a, b in zip(got, both(_unaligned(X), _unaligned(D))):
        np.testing.assert_array_equal(b, a)
    assert gpu_lib.owlgpu_device_status() == 0
