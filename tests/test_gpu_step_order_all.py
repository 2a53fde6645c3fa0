"""Every step kernel that is launched as a dependent of the one before: steps enqueued back to back, in
the stream and in the library's graph, give the bits of the same steps with the stream synchronised
between them.  Sizes whose blocks cover the GPU, so that a step's first blocks start while the one
before still stores its last planes."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu
STEPS, REPEATS = 12, 3


def _heat(n, dtype, sp, graph):
    T, tmp, lam = (N.Field("SVol", n, 1, dtype=dtype) for _ in range(3))
    g = torch.Generator(device="cuda").manual_seed(5)
    T0 = torch.randn(T.tensor.shape, generator=g, device="cuda").to(T.tensor.dtype)
    lam.tensor.uniform_(0.5, 1.0, generator=g)

    def run(apart):
        T.tensor.copy_(T0)
        for _ in range(STEPS if apart else 1):
            N.heat_run(T, tmp, lam, 1 if apart else STEPS, 0.05, sp, use_graph=graph and not apart)
            if apart:
                torch.cuda.synchronize()
        return T.tensor.clone()

    return run


def _transport(n, dtype):
    args = W.transport_inputs(n)

    def run(apart):
        t = N.Transport(*args[:5], n, *args[5:], dtype)
        for _ in range(STEPS if apart else 1):
            t.run(1 if apart else STEPS)
            if apart:
                torch.cuda.synchronize()
        return t.phi.clone()

    return run


def _patches(dtype, graph):
    rng = np.random.default_rng(6)
    shapes = rng.integers(16, 72, size=(96, 3)).astype(np.int32)
    lam = rng.uniform(0.5, 1.5, 96)
    ps = N.PatchSet(shapes, lam, 0.15 / lam, dtype)
    first = torch.randn(ps.arena(0).shape, generator=torch.Generator(device="cuda").manual_seed(7), device="cuda",
                        dtype=torch.float64)

    def run(apart):
        ps.arena(0).copy_(first)
        ps.fill_ghosts(0)
        which = 0
        for _ in range(STEPS if apart else 1):
            which = ps.run(1 if apart else STEPS, start=which, use_graph=graph and not apart)
            if apart:
                torch.cuda.synchronize()
        ps.sync(which)
        return ps.arena(which).clone()

    return run


UNIT, OTHER = (1.0, 1.0, 1.0), (0.5, 0.8, 1.25)


@pytest.mark.parametrize("make", [
    *[pytest.param(lambda n=n, d=d, sp=sp, g=g: _heat(n, d, sp, g), id=f"heat-{d}-{n[0]}-{sp[0]}-{g}")
      for n, d, sp in [((128, 128, 128), "f64", UNIT), ((64, 64, 64), "f64", UNIT), ((150, 131, 98), "f64", OTHER),
                       ((64, 64, 64), "f64", OTHER), ((256, 128, 64), "f32", UNIT), ((323, 197, 60), "f32", UNIT),
                       ((64, 64, 64), "f32", UNIT), ((1030, 90, 20), "f32", UNIT)] for g in (False, True)],
    *[pytest.param(lambda n=n, d=d: _transport(n, d), id=f"transport-{d}-{n}")
      for n, d in [(96, "f64"), (128, "f32"), (126, "f32"), (101, "f32")]],
    *[pytest.param(lambda d=d, g=g: _patches(d, g), id=f"patches-{d}-{g}")
      for d in ("f64", "f32", "f32x2") for g in (False, True)],
])
def test_back_to_back_like_apart(make):
    run = make()
    want = run(True)
    assert torch.isfinite(want).all()
    for _ in range(REPEATS):
        assert torch.equal(run(False), want)
