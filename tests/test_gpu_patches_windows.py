"""nebo_patchset_fill_ghosts and nebo_patchset_sync: FP64 windows get the periodic images of their
interiors, and in FP32 mode the way into the working state and back rounds each value to the nearest
float (subnormal floats, infinities and NaNs included) and fills the window's ghosts."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu
SHAPES = [(2, 2, 2), (3, 5, 4), (31, 4, 3), (96, 7, 5), (127, 3, 4), (129, 5, 3), (1030, 3, 2)]


@pytest.mark.parametrize("dtype,shapes", [("f64", SHAPES), ("f32", SHAPES[:-1]), ("f32", SHAPES)])
def test_windows(dtype, shapes):
    rng = np.random.default_rng(4)
    ps = N.PatchSet(shapes, np.ones(len(shapes)), np.full(len(shapes), 0.1), dtype)
    wins = []
    for p, n in enumerate(shapes):
        a = rng.normal(size=W.window_shape(n, 1)) * 10.0 ** rng.uniform(-47, 20, W.window_shape(n, 1))
        a[1, 1, 1] = np.inf
        a[-2, -2, -2] = np.nan
        wins.append(W.fill_periodic(a.copy(), 1))
        ps.window(0, p).copy_(torch.from_numpy(a))
    ps.fill_ghosts(0)
    for p, w in enumerate(wins):
        assert np.array_equal(ps.window(0, p).cpu().numpy(), w, equal_nan=True)
    ps.arena(0).zero_()
    if dtype == "f64":
        return
    ps.sync(0)
    for p, w in enumerate(wins):
        with np.errstate(over="ignore"):
            want = w.astype(np.float32).astype(np.float64)
        assert np.array_equal(ps.window(0, p).cpu().numpy(), want, equal_nan=True), shapes[p]
