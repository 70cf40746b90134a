"""Workspaces from the library's own stream-ordered pool: calls on several streams
and threads at once, in a captured graph, and of more scratch than the pool keeps
give the results of the same calls made alone."""

import threading

import numpy as np
import pytest

from gpu_util import from_dev

pytestmark = pytest.mark.gpu


def _case(seed, b, ch):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((b, 20, 18, ch), generator=g, device="cuda")
    w = torch.randn((3, 3, ch, ch), generator=g, device="cuda")
    dy = torch.randn((b, 20, 18, ch), generator=g, device="cuda")
    return x, w, dy


def _run(prec, case):
    from owl_gb300.dense import NN, GpuBackend

    nn, (x, w, dy) = NN(GpuBackend(prec)), case
    return (nn.conv2d(x, w, [1, 1]), nn.conv2d_backward_input(x, w, [1, 1], dy),
            nn.conv2d_backward_kernel(x, w, [1, 1], dy))


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
def test_threads_and_streams(gpu_lib, prec):
    import torch

    cases = [_case(s, 2 + s, 32 * (1 + s % 2)) for s in range(4)]
    alone = [[from_dev(t) for t in _run(prec, c)] for c in cases]
    got, errs = [None] * 4, []

    def work(i):
        try:
            s = torch.cuda.Stream()
            s.wait_stream(torch.cuda.default_stream())
            with torch.cuda.stream(s):
                for _ in range(20):
                    got[i] = _run(prec, cases[i])
            s.synchronize()
        except Exception as e:  # reported below, by the test's own thread
            errs.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errs
    for a, g in zip(alone, got):
        for u, v in zip(a, g):
            np.testing.assert_array_equal(from_dev(v), u)


def test_captured_and_large_scratch(gpu_lib):
    import torch

    case = _case(9, 3, 64)
    ref = [from_dev(t) for t in _run("bf16", case)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _run("bf16", case)
    # between replays: partials of 64 M elements (256 MB of scratch and more)
    from owl_gb300.dense import NN, GpuBackend
    from owl_gb300.layers import Layers

    L = Layers(NN(GpuBackend("bf16")))
    a = torch.ones((4096, 64), device="cuda")
    b = torch.ones((4096, 4096), device="cuda")
    for _ in range(2):
        graph.replay()
        c = L.dot(a, b, trans_a=True)
        torch.cuda.synchronize()
    np.testing.assert_array_equal(from_dev(c), np.full((64, 4096), 4096.0, np.float32))
    for u, v in zip(ref, out):
        np.testing.assert_array_equal(from_dev(v), u)
