"""Long sums in split BF16 against float64, at the mode's tolerance: <= 1e-5 of the
largest element.  The tensor core rounds an accumulator toward zero at every MMA, so
the error grows with the MMAs that one takes in turn; these are layers of many pixels
and wide blocks, and products of long inner dimensions."""

import pytest

from gpu_util import from_dev, rel

pytestmark = pytest.mark.gpu


def _draw(seed, *shapes):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(s, generator=g, device="cuda") for s in shapes]


# batch, rows, columns, channels in and out, kernel
WGRAD = [
    (64, 7, 7, 512, 512, 3),
    (64, 14, 14, 512, 512, 3),
    (4, 56, 56, 512, 512, 3),
    (32, 14, 14, 1024, 256, 1),
]


@pytest.mark.parametrize("b,h,w,ci,co,k", WGRAD)
def test_weight_gradient(gpu_lib, b, h, w, ci, co, k):
    import torch

    from owl_gb300.dense import NN, GpuBackend

    x, dy, kern = _draw(ci, (b, h, w, ci), (b, h, w, co), (k, k, ci, co))
    got = NN(GpuBackend("bf16x3")).conv2d_backward_kernel(x, kern, [1, 1], dy)
    assert gpu_lib.owlgpu_last_conv_path() == 1
    p = k // 2
    xp = torch.nn.functional.pad(x.double(), (0, 0, p, p, p, p))
    d = dy.double().reshape(-1, co)
    ref = torch.stack([xp[:, i:i + h, j:j + w].reshape(-1, ci).T @ d
                       for i in range(k) for j in range(k)]).reshape(got.shape)
    assert rel(from_dev(got), from_dev(ref)) <= 1e-5


@pytest.mark.parametrize("m,n,k", [(2048, 2048, 16384), (1024, 1024, 65536), (512, 1024, 3136)])
def test_dense_product(gpu_lib, m, n, k):
    from owl_gb300.dense import NN, GpuBackend
    from owl_gb300.layers import Layers

    a, b = _draw(m + n, (k, m), (k, n))
    got = Layers(NN(GpuBackend("bf16x3"))).dot(a, b, trans_a=True)
    assert rel(from_dev(got), from_dev(a.double().T @ b.double())) <= 1e-5
