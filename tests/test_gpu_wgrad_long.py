"""The weight gradient of a long 1-D signal: planning it takes no time that grows with
its length, and the result is exact (operands of small whole numbers, sums below 2^24)."""

import time

import pytest

pytestmark = pytest.mark.gpu


def test_long_signal(gpu_lib):
    import torch

    from owl_gb300.dense import NN, GpuBackend

    n = 1 << 28
    x = torch.zeros((1, n, 1, 1), device="cuda")
    dy = torch.zeros((1, n, 1, 1), device="cuda")
    x[:, ::4096] = 3.0
    dy[:, ::2048] = 2.0
    w = torch.zeros((3, 1, 1, 1), device="cuda")
    nn = NN(GpuBackend("bf16"))
    best = 1.0
    for _ in range(4):
        torch.cuda.synchronize()
        t = time.perf_counter()
        dw = nn.conv2d_backward_kernel(x, w, [1, 1], dy)
        best = min(best, time.perf_counter() - t)
    assert gpu_lib.owlgpu_last_conv_path() == 1
    assert dw.flatten().tolist() == [0.0, 6.0 * (n // 4096), 0.0]
    # the call returns when the work is queued: some 20 us (2^28 / 8 steps of a search
    # over tile counts took 70 ms and more)
    assert best < 0.01
