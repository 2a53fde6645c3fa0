"""ParticleToCell's fold and both directions' face tables where they can go wrong: slices of 0 to
several hundred entries per cell (below, at and beyond the fold's staging capacity of 512), a window
whose edges exceed the shared-memory table, boxes wider than 4 cells; bit-identical to the oracle."""
import numpy as np
import pytest
import torch

import oracle_dsl as O
import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _check(pc, n, g):
    want_c2p, want_p2c = O.particle_ops(pc)
    cell = N.Field("SVol", n, g, tensor=torch.from_numpy(pc["cell"]).cuda())
    pos = [torch.from_numpy(pc[k]).cuda() for k in ("px", "py", "pz")]
    size, val = torch.from_numpy(pc["psize"]).cuda(), torch.from_numpy(pc["pval"]).cuda()
    out = torch.empty(len(pc["px"]), dtype=torch.float64, device="cuda")
    N.cell_to_particle(cell, *pos, size, out, pc["spacing"], pc["low"])
    dest = N.Field("SVol", n, g)
    N.particle_to_cell(val, *pos, size, dest, pc["spacing"], pc["low"])
    assert np.array_equal(out.cpu().numpy().view(np.uint64), want_c2p.view(np.uint64))
    assert np.array_equal(dest.numpy().view(np.uint64), want_p2c.view(np.uint64))


@pytest.mark.parametrize("per_cell", [0.05, 1, 20, 60, 130])
def test_slice_lengths(per_cell):
    n = (6, 5, 4)
    m = int(per_cell * 6 * 5 * 4) + 1
    _check(W.particle_inputs(n, 1, m, size_range=(0.3, 2.5), seed=m), n, 1)


@pytest.mark.parametrize("m", [511, 512, 513, 700])
def test_one_long_slice(m):
    # every particle inside one cell: its slice holds m entries
    n = (8, 8, 8)
    pc = W.particle_inputs(n, 1, m, size_range=(0.1, 0.2), seed=3)
    for k in ("px", "py", "pz"):
        pc[k] = 3.5 + np.random.default_rng(len(k) + m).uniform(0.2, 0.8, m) * 0.5
    _check(pc, n, 1)


def test_window_beyond_the_table():
    n = (1020, 3, 2)
    _check(W.particle_inputs(n, 1, 4000, size_range=(0.3, 2.5), seed=5), n, 1)


def test_wide_boxes():
    n = (40, 12, 9)
    _check(W.particle_inputs(n, 1, 700, size_range=(0.5, 7.5), seed=8), n, 1)
