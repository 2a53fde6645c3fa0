"""FP32 heat steps bit for bit against their operations restated in numpy float32: windows with an
even pitch and 8-byte aligned rows round every flux, the others take the high x flux and, in every
fourth row, the low y flux unrounded.  Widths on either side of each kernel's range."""
import numpy as np
import pytest
import torch

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32, F64 = np.float32, np.float64


def _fma(a, b, c):
    """RN32(a b + c): the product is exact in 64 bits; the sum is rounded to odd there, then to 32 bits."""
    p, c = a.astype(F64) * b.astype(F64), c.astype(F64)
    s = p + c
    t = s - p
    e = (p - (s - t)) + (c - t)  # s + e = p + c exactly
    i = s.view(np.int64)
    i = np.where((e != 0) & (i & 1 == 0), np.where((e > 0) == (s > 0), i + 1, i - 1), i)
    return i.view(F64).astype(F32)


def _step(T, L, w, paired):
    c = (slice(1, -1),) * 3
    v = T[c]
    for k, ax in enumerate((2, 1, 0)):
        lo, hi = list(c), list(c)
        lo[ax], hi[ax] = slice(0, -2), slice(2, None)
        sl, dl = L[tuple(lo)] + L[c], T[c] - T[tuple(lo)]
        sh, dh = L[c] + L[tuple(hi)], T[tuple(hi)] - T[c]
        d = sh * dh - sl * dl
        if not paired and k == 0:
            d = _fma(sh, dh, -(sl * dl))
        if not paired and k == 1:
            d[:, ::4] = _fma(-sl, dl, sh * dh)[:, ::4]
        v = _fma(d, np.full_like(d, w[k]), v)
    return v


def _field(a, off):
    """An FP32 field whose allocation starts `off` floats after a 512-byte boundary."""
    flat = torch.empty(a.size + off, dtype=torch.float32, device="cuda")
    t = flat[off:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return N.Field("SVol", tuple(d - 2 for d in a.shape[::-1]), 1, dtype="f32", tensor=t)


@pytest.mark.parametrize("offs", [(0, 0), (1, 3), (2, 0)])
@pytest.mark.parametrize("n", [(2, 2, 2), (3, 5, 4), (64, 24, 9), (192, 9, 7), (193, 8, 7), (200, 16, 5), (254, 7, 6),
                               (256, 8, 5), (323, 13, 6), (1024, 6, 4), (1029, 38, 6), (1030, 9, 6)])
def test_step_bits(n, offs):
    rng = np.random.default_rng(11)
    shp = W.window_shape(n, 1)
    L = W.fill_periodic(rng.uniform(0.5, 1.5, shp).astype(F32), 1)
    T = W.fill_periodic(rng.normal(size=shp).astype(F32), 1)
    dt, sp = 0.1, (0.9, 1.1, 1.3)
    out = _field(np.zeros_like(T), 0)
    N.heat_step(_field(T, offs[0]), out, _field(L, offs[1]), dt, sp)
    w = [F32(0.5 * dt / (d * d)) for d in sp]
    paired = n[0] % 2 == 0 and offs[0] % 2 == 0 and offs[1] % 2 == 0
    want = _step(T, L, w, paired)
    assert (out.numpy()[1:-1, 1:-1, 1:-1].view(np.uint32) == want.view(np.uint32)).all()
