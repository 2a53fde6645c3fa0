"""FP32 patches on the slab layout, four cells of a row to a thread: rows that end inside a quad, rows
of one quad and of a whole strip, strips with fewer rows than the others and one-plane-deep sets.

The reference does the step in numpy float32 with the kernel's order of sums; its fused
multiply-adds are formed in double and rounded once more, which may move a result by one unit.
With |T| <= 1 and k <= 1/6 a step's two such units are at most 2^-23 (1 + 12 k) <= 2^-21 and the step
itself does not amplify, so n steps stay within n 2^-21."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu
SHAPES = [(2, 2, 2), (3, 5, 4), (4, 300, 2), (5, 7, 9), (31, 40, 3), (64, 17, 70), (65, 16, 5), (96, 11, 4),
          (127, 9, 3), (1021, 3, 2), (1024, 2, 3)]


def step(T, k):
    T, k = T.astype(np.float32), float(np.float32(k))
    s = [np.roll(T, d, ax) for ax in (2, 1, 0) for d in (1, -1)]
    nb = ((s[0] + s[1]) + (s[2] + s[3])) + (s[4] + s[5])
    lap = (-6.0 * T.astype(np.float64) + nb).astype(np.float32)
    return (k * lap.astype(np.float64) + T).astype(np.float32)


@pytest.mark.parametrize("steps", [1, 5])
def test_f32_quads(steps):
    rng = np.random.default_rng(steps)
    lam = rng.uniform(0.3, 0.8, len(SHAPES))
    dt = rng.uniform(0.05, 0.2, len(SHAPES))
    ps = N.PatchSet(SHAPES, lam, dt, "f32")
    want = []
    for p, n in enumerate(SHAPES):
        T = rng.uniform(-1.0, 1.0, n[::-1]).astype(np.float32)
        w = np.zeros(W.window_shape(n, 1))
        w[1:-1, 1:-1, 1:-1] = T
        ps.window(0, p).copy_(torch.from_numpy(W.fill_periodic(w, 1)))
        for _ in range(steps):
            T = step(T, 0.5 * dt[p] * (lam[p] + lam[p]))
        want.append(T)
    ps.fill_ghosts(0)
    cur = ps.run(steps)
    ps.sync(cur)
    for p in range(len(SHAPES)):
        got = ps.window(cur, p).cpu().numpy()[1:-1, 1:-1, 1:-1]
        assert np.abs(got - want[p]).max() <= steps * 2.0**-21, SHAPES[p]
