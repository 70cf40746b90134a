"""What the library's scratch pool keeps: a call's workspace stays reserved up to
256 MB, what is above goes back at the next synchronisation, owlgpu_trim gives back
the rest, and calls after it, captured graphs among them, give the same results.
Seen in the device's free memory, with the workspace (the kernel tensor's image,
taps x channels x channels x 2 bytes) larger than the drift allowed for."""

import numpy as np
import pytest

from gpu_util import from_dev

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    import torch

    return torch.cuda.mem_get_info()[0]


def _conv(ci, co):
    """A small convolution with a large kernel tensor, warmed up so that its output's
    memory is in the framework's cache."""
    import torch

    from owl_gb300.dense import NN, GpuBackend

    g = torch.Generator(device="cuda").manual_seed(ci)
    x = torch.randn((1, 4, 4, ci), generator=g, device="cuda")
    w = torch.randn((3, 3, ci, co), generator=g, device="cuda")
    nn = NN(GpuBackend("bf16"))
    return (lambda: nn.conv2d(x, w, [1, 1])), from_dev(nn.conv2d(x, w, [1, 1]))


def test_trim_gives_scratch_back(gpu_lib):
    import torch

    image = 9 * 2048 * 4096 * 2  # 151 MB: below what the pool keeps
    call, ref = _conv(2048, 4096)
    assert gpu_lib.owlgpu_trim() == 0
    before = _free()
    y = call()
    torch.cuda.synchronize()
    assert before - _free() >= image - 16 * MB  # kept across the synchronisation
    assert gpu_lib.owlgpu_trim() == 0
    assert before - _free() <= 16 * MB
    np.testing.assert_array_equal(from_dev(y), ref)
    np.testing.assert_array_equal(from_dev(call()), ref)


def test_large_scratch_goes_back(gpu_lib):
    import torch

    image = 9 * 4096 * 4096 * 2  # 302 MB: above it
    small, ref_small = _conv(64, 128)
    call, ref = _conv(4096, 4096)
    assert gpu_lib.owlgpu_trim() == 0
    before = _free()
    y = call()
    assert before - _free() >= image - 16 * MB  # reserved at the launch
    torch.cuda.synchronize()
    assert before - _free() <= 256 * MB
    np.testing.assert_array_equal(from_dev(y), ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = small()
    for _ in range(2):  # replays around workspaces that come and go
        graph.replay()
        np.testing.assert_array_equal(from_dev(call()), ref)
        assert gpu_lib.owlgpu_trim() == 0
        graph.replay()
        np.testing.assert_array_equal(from_dev(out), ref_small)
