"""The FP64 patch step (integer face fluxes) against nebo_heat_step on each patch with its lambda as a
constant field: identical bits for every tile width, at remainders in x, y and z, and for values the
integer flux leaves to the FP64 unit (NaNs count as equal whatever their payload)."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu
SHAPES = [(2, 2, 2), (16, 16, 16), (15, 17, 18), (17, 9, 33), (32, 8, 16), (40, 7, 5), (41, 5, 17), (64, 4, 3),
          (65, 13, 34), (96, 96, 20)]


@pytest.mark.parametrize("tune", [False, True])
@pytest.mark.parametrize("kind", ["smooth", "special"])
def test_patch_steps(kind, tune):
    rng = np.random.default_rng(9)
    lam = rng.uniform(0.5, 1.5, len(SHAPES))
    dt = 0.15 / lam
    ps = N.PatchSet(SHAPES, lam, dt, "f64")
    if tune:
        ps.autotune()
    wins = []
    for p, n in enumerate(SHAPES):
        shp = W.window_shape(n, 1)
        T = W.gaussian_bump(n, 1, sigma=min(n) / 3.0) + rng.normal(0, 1e-3, shp)
        if kind == "special":
            T *= 10.0 ** rng.uniform(-200, 200, shp)
            T[rng.random(shp) < 0.1] = -0.0
            T[rng.random(shp) < 0.1] = 5e-324
            T[tuple(s // 2 for s in shp)] = np.inf
            T[1, 1, 1] = np.nan
        wins.append(W.fill_periodic(T, 1))
        ps.window(0, p).copy_(torch.from_numpy(wins[p]))
    ps.fill_ghosts(0)
    steps = 3
    which = ps.run(steps)
    for p, n in enumerate(SHAPES):
        f = [N.Field.from_numpy("SVol", wins[p], 1), N.Field("SVol", n, 1)]
        L = N.Field.from_numpy("SVol", np.full(wins[p].shape, lam[p]), 1)
        for k in range(steps):
            N.heat_step(f[k & 1], f[(k + 1) & 1], L, float(dt[p]))
        want, got = f[steps & 1].numpy(), ps.window(which, p).cpu().numpy()
        same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
        assert same.all(), (n, int((~same).sum()))
