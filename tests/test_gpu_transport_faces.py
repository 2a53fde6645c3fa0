"""The FP64 transport run on precomputed face coefficients (two or more steps) against the same steps
one call at a time, which form the coefficients in every stage, and against a run that the caller
records into a graph: the coefficients are the same operations, so the bits are equal.  Sizes at
tile edges and remainders; each also within 1e-13 of the oracle's run."""
import numpy as np
import pytest
import torch

import oracle_dsl as O
import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 5, 8, 31, 32, 33, 41])
def test_coefficients_once_or_every_stage(n):
    phi, u, v, w, lam, dt, nu = W.transport_inputs(n)
    make = lambda: N.Transport(phi, u, v, w, lam, n, dt, nu, "f64")  # noqa: E731
    a, b, c = make(), make(), make()
    a.run(3)
    for _ in range(3):
        b.run(1)
    assert torch.equal(a.phi, b.phi)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        c.run(3)
    c.phi.copy_(torch.from_numpy(phi))
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(a.phi, c.phi)
    ref = O.transport_run(phi, u, v, w, lam, n, 3, dt, nu)
    assert np.abs(a.phi.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
