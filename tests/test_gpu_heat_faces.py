"""nebo_heat_run on precomputed face coefficients (three or more exact FP64 steps) against the same
steps taken one nebo_heat_step at a time: identical bits, at the tiles' edges and remainders, for
values whose fluxes the integer form does not cover (infinities, NaNs, -0, subnormals, huge and tiny
magnitudes) and for coefficients of any sign; NaNs count as equal whatever their payload."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _inputs(n, kind):
    rng = np.random.default_rng(5)
    shp = W.window_shape(n, 1)
    lam = rng.uniform(0.5, 1.5, shp)
    T = W.gaussian_bump(n, 1, sigma=4.0) + rng.normal(0.0, 1e-3, shp)
    if kind == "wide":
        T = rng.normal(size=shp) * 10.0 ** rng.uniform(-300, 290, shp)
        lam = rng.normal(size=shp) * 10.0 ** rng.uniform(-20, 2, shp)
    elif kind == "special":
        pick = rng.random(shp)
        for lo, v in ((0.0, 0.0), (0.05, -0.0), (0.1, 5e-324), (0.12, -3e-310), (0.14, 1.7e308)):
            T[(pick >= lo) & (pick < lo + 0.02)] = v
        lam[rng.random(shp) < 0.03] = 0.0
        lam[rng.random(shp) < 0.02] = 4e-310
        at = tuple(s // 2 for s in shp)
        T[at] = np.inf
        T[1, 1, 1] = np.nan
    elif kind == "flat":
        T[:] = 1.0 + rng.integers(0, 3, shp) * 2.0 ** -52
    return W.fill_periodic(lam, 1), W.fill_periodic(T, 1)


@pytest.mark.parametrize("sp", [(1.0, 1.0, 1.0), (0.5, 0.8, 1.25)])
@pytest.mark.parametrize("kind", ["smooth", "wide", "special", "flat"])
@pytest.mark.parametrize("n", [(2, 2, 2), (31, 7, 5), (32, 8, 4), (33, 9, 7), (64, 16, 3), (97, 25, 40)])
def test_run_equals_single_steps(n, kind, sp):
    lam, T0 = _inputs(n, kind)
    steps, dt = 5, 0.04
    L = N.Field.from_numpy("SVol", lam, 1)
    ref = [N.Field.from_numpy("SVol", T0, 1), N.Field("SVol", n, 1)]
    for k in range(steps):
        N.heat_step(ref[k & 1], ref[(k + 1) & 1], L, dt, sp)
    want = ref[steps & 1].numpy()
    for graph in (False, True):
        T, tmp = N.Field.from_numpy("SVol", T0, 1), N.Field("SVol", n, 1)
        N.heat_run(T, tmp, L, steps, dt, sp, use_graph=graph)
        got = T.numpy()
        same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
        assert same.all(), (graph, int((~same).sum()))


def test_run_inside_a_callers_capture():
    # a stream that the caller records takes the form without scratch: no allocation nodes
    n, steps, dt = (40, 24, 12), 4, 0.04
    lam, T0 = _inputs(n, "smooth")
    L = N.Field.from_numpy("SVol", lam, 1)
    T, tmp = N.Field.from_numpy("SVol", T0, 1), N.Field("SVol", n, 1)
    N.heat_run(T, tmp, L, steps, dt, use_graph=False)
    want = T.numpy()
    T.tensor.copy_(torch.from_numpy(T0))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        N.heat_run(T, tmp, L, steps, dt, use_graph=False)
    T.tensor.copy_(torch.from_numpy(T0))
    g.replay()
    torch.cuda.synchronize()
    assert (T.numpy().view(np.uint64) == want.view(np.uint64)).all()
