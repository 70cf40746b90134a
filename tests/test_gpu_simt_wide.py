"""Dense products on the CUDA cores of more columns than 65535 tiles of 32 or of 64
hold (a grid's y axis takes no more tiles), in float32 and float64 and in every
transposition: operands of small whole numbers, so every element is exact."""

import pytest

pytestmark = pytest.mark.gpu

# rows, columns, depth; a or b transposed
CASES = [
    ("float32", 1, 2_200_000, 16, False, False),
    ("float32", 5, 2_200_000, 16, False, True),
    ("float32", 4, 2_200_001, 7, False, False),     # scalar kernel
    ("float32", 4, 2_200_000, 32, True, False),
    ("float32", 3, 2_200_000, 16, True, False),
    ("float32", 100, 4_300_000, 16, False, False),  # more than 65535 tiles of 64
    ("float32", 2, 4_300_000, 16, False, True),
    ("float32", 16, 4_300_000, 20, True, False),
    ("float64", 1, 2_200_000, 16, False, False),
    ("float64", 17, 2_200_000, 3, False, True),
    ("float64", 9, 2_200_000, 5, True, False),
]


@pytest.mark.parametrize("kind,m,n,k,ta,tb", CASES)
def test_wide_products(gpu_lib, kind, m, n, k, ta, tb):
    import torch

    from owl_gb300.dense import NN, GpuBackend
    from owl_gb300.layers import Layers

    L = Layers(NN(GpuBackend("fp32")))
    dt = getattr(torch, kind)
    g = torch.Generator(device="cuda").manual_seed(m + n + k)

    def whole(*shape):
        return torch.randint(-3, 4, shape, generator=g, device="cuda").to(dt)

    a = whole(k, m) if ta else whole(m, k)
    b = whole(n, k) if tb else whole(k, n)
    c = L.dot(a, b, trans_a=ta, trans_b=tb)
    A, B = (a.T if ta else a).double(), (b.T if tb else b)
    for n0 in range(0, n, 1 << 20):
        n1 = min(n, n0 + (1 << 20))
        assert torch.equal(c[:, n0:n1].double(), A @ B[:, n0:n1].double())
