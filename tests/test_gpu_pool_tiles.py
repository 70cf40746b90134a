"""Pooling at the edges of its tiles, bit for bit against the oracle: the
overlapping backward's blocks of input elements (partial tiles, one-element
axes, channel runs that do not fill a block, windows wider than a tile, windows
with too many taps for the tiled kernel) and the fixed-window forward's clipped
windows."""

import numpy as np
import pytest

import oracle
from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu

# input dims, channels, window, stride
CASES_2D = [
    ((17, 16), 64, (3, 3), (2, 2)), ((1, 33), 4, (3, 3), (1, 1)), ((15, 31), 68, (3, 2), (1, 1)),
    ((9, 7), 3, (3, 3), (2, 2)), ((40, 18), 12, (5, 7), (2, 3)), ((18, 17), 8, (17, 18), (1, 1)),
    ((33, 9), 130, (3, 3), (3, 1)), ((16, 16), 4, (2, 5), (3, 2)), ((7, 7), 256, (2, 2), (1, 1)),
    ((112, 5), 16, (3, 3), (2, 2)), ((11, 13), 5, (3, 3), (3, 3)), ((17, 31), 68, (3, 3), (1, 1)),
    ((35, 64), 132, (3, 3), (2, 2)), ((2, 33), 4, (2, 2), (1, 1)),
]
CASES_3D = [
    ((9, 8, 7), 16, (3, 3, 3), (2, 2, 2)), ((5, 1, 17), 3, (2, 2, 2), (1, 1, 1)),
    ((8, 9, 10), 66, (3, 2, 4), (2, 1, 3)), ((7, 7, 7), 4, (7, 7, 6), (1, 1, 1)),
    ((6, 5, 9), 4, (2, 2, 2), (2, 2, 2)), ((17, 9, 10), 68, (3, 3, 3), (2, 2, 2)),
    ((3, 16, 1), 8, (3, 3, 3), (2, 2, 2)),
]


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64])
@pytest.mark.parametrize("padding", ["SAME", "VALID"])
@pytest.mark.parametrize("dims,ch,win,stride", CASES_2D + CASES_3D)
def test_pool_tiles(dims, ch, win, stride, padding, dtype):
    from owl_gb300.dense import NN, GpuBackend

    if padding == "VALID" and any(k > n for k, n in zip(win, dims)):
        pytest.skip("window larger than the input")
    G, O = NN(GpuBackend("fp32")), NN(oracle.OracleBackend())
    rng = np.random.default_rng(len(dims) * 100 + ch)

    def draw(shape):
        # few distinct values: ties decide which element wins
        a = rng.integers(-3, 4, shape).astype(np.float64) / 4
        if np.issubdtype(dtype, np.complexfloating):
            a = a + 1j * rng.integers(-3, 4, shape) / 4
        return a.astype(dtype)

    x = draw((2, *dims, ch))
    if not np.issubdtype(dtype, np.complexfloating):
        x[0, 0] = -np.inf  # some windows select nothing
        x[1, -1, ..., -1] = np.nan
        x[1, 0, ..., 0] = np.inf
    nd = f"{len(dims)}d"
    for mode in ("max", "avg"):
        fwd, bwd = f"{mode}_pool{nd}", f"{mode}_pool{nd}_backward"
        y = getattr(O, fwd)(x, list(win), list(stride), padding)
        yd = getattr(G, fwd)(to_dev(x), list(win), list(stride), padding)
        np.testing.assert_array_equal(from_dev(yd), y)
        dy = (rng.standard_normal(y.shape) * (1 + np.arange(y.shape[-1]))).astype(dtype)
        dx = getattr(O, bwd)(padding, x, list(win), list(stride), dy)
        dxd = getattr(G, bwd)(padding, to_dev(x), list(win), list(stride), to_dev(dy))
        np.testing.assert_array_equal(from_dev(dxd), dx)
