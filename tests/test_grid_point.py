"""The P(t) grid point nearest to a branch length: the kernels place t on the logarithmic grid in FP32
and let an FP64 comparison with the next point decide.  Restated here against the same rule with the
place in FP64, at and around every grid point and midpoint (whole numbers: no tolerance)."""
import numpy as np


def _nearest(place, t, grid):
    g = np.clip(np.floor(place).astype(np.int64), 0, len(grid) - 1)
    nxt = np.minimum(g + 1, len(grid) - 1)
    return np.where((g + 1 < len(grid)) & (grid[nxt] - t < t - grid[g]), nxt, g)


def test_fp32_place_gives_the_same_point():
    lr = np.log(1.002)
    grid = 1e-5 * np.exp(lr * np.arange(6500))
    mid = 0.5 * (grid[1:] + grid[:-1])
    rel = np.array([0.0, 1e-16, 1e-13, 1e-10, 1e-8, 1e-7, 1e-6, 1e-5, 3e-4])
    t = np.concatenate([np.outer(x, np.concatenate([1.0 + rel, 1.0 - rel])).ravel() for x in (grid, mid)])
    t = t[t >= grid[0]]
    f64 = _nearest(np.log(t / grid[0]) / lr, t, grid)
    f32 = np.log(t.astype(np.float32) / np.float32(grid[0])) / np.float32(lr)
    for ulps in (-4, 0, 4):           # the device's logarithm and division may round otherwise
        place = f32 * np.float32(1.0 + ulps * 2.0 ** -24)
        assert np.array_equal(_nearest(place, t, grid), f64)
