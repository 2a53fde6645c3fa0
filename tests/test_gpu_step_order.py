"""Step kernels launched as dependents of one another read nothing of the step before ahead of its end:
runs of the same inputs give the same bits every time, at sizes whose blocks cover the GPU in one wave
(the next step's blocks then start while the last planes are still being written)."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _gradient(rng, n):
    shp = W.window_shape((n, n, n), 1)
    F = lambda a: N.Field.from_numpy("SVol", W.fill_periodic(a, 1), 1)  # noqa: E731
    T, lam, target = F(rng.normal(size=shp)), F(rng.uniform(0.5, 1.0, shp)), F(rng.normal(size=shp))

    def run():
        J, gT, gl = N.heat_gradient(T, lam, target, 48, 0.1)
        return [torch.tensor(float(J)), gT.tensor.clone(), gl.tensor.clone()]

    return run


def _transport(rng, n):
    phi, u, v, w, lam, dt, nu = W.transport_inputs(n)

    def run():
        t = N.Transport(phi, u, v, w, lam, n, dt, nu, "f64")
        t.run(10)
        return [t.phi.clone()]

    return run


@pytest.mark.parametrize("make,n", [(_gradient, 128), (_gradient, 96), (_transport, 96)])
def test_same_bits_every_run(make, n):
    run = make(np.random.default_rng(8), n)
    first = run()
    for _ in range(12):
        assert all(torch.equal(a, b) for a, b in zip(first, run()))
