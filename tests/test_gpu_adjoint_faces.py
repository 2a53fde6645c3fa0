"""The reverse steps of nebo_heat_gradient (integer differences on precomputed face coefficients)
against nebo_heat_adjoint_step along the same FP64 trajectory: identical dJ/dT0 and dJ/dlambda, at the
tiles' edges and remainders and for values the integer difference leaves to the FP64 unit.  With FP32
products or an FP32 forward the gradient stays within the documented 1e-5."""
import numpy as np
import pytest

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["smooth", "wide"])
@pytest.mark.parametrize("n", [(2, 2, 2), (31, 7, 5), (32, 8, 4), (33, 9, 7), (64, 16, 3), (70, 25, 21)])
def test_gradient_equals_single_steps(n, kind):
    rng = np.random.default_rng(6)
    shp = W.window_shape(n, 1)
    lam = W.fill_periodic(rng.uniform(0.5, 1.5, shp), 1)
    T = rng.normal(size=shp)
    if kind == "wide":
        T *= 10.0 ** rng.uniform(-150, 0, shp)
        T[rng.random(shp) < 0.1] = -0.0
        T[rng.random(shp) < 0.1] = 5e-324
    T0, target = W.fill_periodic(T, 1), W.fill_periodic(rng.normal(size=shp), 1)
    steps, dt = 6, 0.1
    F = lambda a: N.Field.from_numpy("SVol", a, 1)  # noqa: E731
    L = F(lam)
    J, gT, gl = N.heat_gradient(F(T0), L, F(target), steps, dt)
    states = [F(T0)]
    for _ in range(steps):
        states.append(N.Field("SVol", n, 1))
        N.heat_step(states[-2], states[-1], L, dt)
    A, B, g = N.Field("SVol", n, 1), N.Field("SVol", n, 1), N.Field("SVol", n, 1)
    A.tensor.copy_(states[-1].tensor - F(target).tensor)
    for k in reversed(range(steps)):
        N.heat_adjoint_step(states[k], A, B, L, g, dt)
        A, B = B, A
    inner = (slice(1, -1),) * 3
    assert (gT.numpy().view(np.uint64) == A.numpy().view(np.uint64)).all()
    assert (gl.numpy()[inner] == g.numpy()[inner]).all()
    for kw in (dict(products="f32"), dict(forward="f32"), dict(products="f32", forward="f32")):
        if kind == "wide":
            continue
        J2, gT2, gl2 = N.heat_gradient(F(T0), L, F(target), steps, dt, **kw)
        for a, b in ((gT2, gT), (gl2, gl)):
            assert np.abs(a.numpy() - b.numpy()).max() <= 1e-5 * np.abs(b.numpy()).max(), kw
