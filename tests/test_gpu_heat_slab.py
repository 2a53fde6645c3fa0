"""One FP32 nebo_heat_step on slabs of any row pitch and alignment, against the FP64 step on the same
(widened) inputs: within 16 * 2^-24 of max|T| per cell (each of the six fluxes is at most
0.075 * 3 * 2 max|T| in weight and goes through four FP32 roundings, the sums through four more).
Ghost cells equal their interior images bit for bit."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _field(a, off):
    """An FP32 field whose allocation starts `off` floats after a 512-byte boundary."""
    flat = torch.empty(a.size + off, dtype=torch.float32, device="cuda")
    t = flat[off:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    n = tuple(d - 2 for d in a.shape[::-1])
    return N.Field("SVol", n, 1, dtype="f32", tensor=t)


@pytest.mark.parametrize("offs", [(0, 0, 0), (1, 3, 2)])
@pytest.mark.parametrize("n", [(2, 2, 2), (3, 5, 4), (31, 4, 3), (32, 9, 7), (33, 8, 10), (65, 6, 5), (193, 7, 9),
                               (256, 16, 5), (255, 21, 4), (323, 5, 6), (1023, 4, 3), (1024, 5, 4), (1029, 7, 6),
                               (1030, 8, 6)])
def test_fp32_step(n, offs):
    rng = np.random.default_rng(3)
    shp = W.window_shape(n, 1)
    lam = W.fill_periodic(rng.uniform(0.5, 1.5, shp).astype(np.float32), 1)
    T0 = W.fill_periodic(rng.normal(size=shp).astype(np.float32), 1)
    out = _field(np.full(shp, np.nan, np.float32), offs[2])
    N.heat_step(_field(T0, offs[0]), out, _field(lam, offs[1]), 0.15 / 1.5)
    ref = N.Field("SVol", n, 1)
    N.heat_step(N.Field.from_numpy("SVol", T0.astype(np.float64), 1), ref,
                N.Field.from_numpy("SVol", lam.astype(np.float64), 1), float(np.float32(0.15 / 1.5)))
    got, want = out.numpy(), ref.numpy()
    assert np.abs(got - want).max() <= 16 * 2.0 ** -24 * np.abs(T0).max()
    assert (got.view(np.uint32) == W.fill_periodic(got.copy(), 1).view(np.uint32)).all()
