"""nebo_reduce (one launch), nebo_reduce_async (two) and nebo_reduce_all on the walks and sizes where
they can go wrong: one-run and row-wise regions, remainders of a batch and of a block, several
blocks, sums at the ends of the exponent range, zeros, cancellation, infinities and NaNs, and calls
from several threads at once.  A sum must be within 2^-51 of the sum of magnitudes of math.fsum's
value (three FP64 roundings in a batch of 8, exact beyond), a norm within 2^-51 relative."""
import math
import threading

import numpy as np
import pytest
import torch

import spatialops_gb300 as N

pytestmark = pytest.mark.gpu


def _check(a, ghost, dtype="f64", scale=1.0):
    f = N.Field.from_numpy("SVol", a, ghost, dtype=dtype)
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    one = torch.zeros(1, dtype=torch.float64, device="cuda")
    for interior in (False, True):
        r = a[ghost:-ghost, ghost:-ghost, ghost:-ghost] if interior and ghost else a
        v = r.reshape(-1).astype(np.float64)
        want = {"sum": math.fsum(v), "max": v.max(), "min": v.min(),
                "norm": math.sqrt(math.fsum((v / scale) ** 2)) * scale}
        tol = {"sum": 2.0 ** -51 * math.fsum(np.abs(v)), "max": 0.0, "min": 0.0, "norm": 2.0 ** -51 * want["norm"]}
        N.reduce_all(f, interior, out)
        allr = dict(zip(("sum", "max", "min", "norm"), out.tolist()))
        for op in want:
            N.reduce_async(f, op, interior, one)
            for got in (N._reduce(f, op, interior), one.item(), allr[op]):
                if op == "norm" and want["norm"] > 1.3e154:  # its square leaves the doubles
                    assert not math.isfinite(got)
                    continue
                assert abs(got - want[op]) <= tol[op], (op, interior, got, want[op])


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(4, 4, 4), (4, 5, 6), (4, 5, 230), (9, 11, 21), (5, 40, 259), (70, 66, 64),
                                   (130, 131, 133)])
def test_regions(shape, dtype):
    a = np.random.default_rng(1).normal(size=shape)
    if dtype == "f32":
        a = a.astype(np.float32).astype(np.float64)
    _check(a, 1, dtype)


@pytest.mark.parametrize("scale", [1e-150, 1e150])
def test_scales_and_cancellation(scale):
    rng = np.random.default_rng(2)
    a = rng.normal(size=(20, 21, 22)) * scale
    a[::2] *= 1e9
    a[1::2, ::3] = -a[1::2, ::3]
    _check(a, 1, scale=scale)


def test_ends_of_the_exponent_range_and_zeros():
    a = np.random.default_rng(3).uniform(-1, 1, (12, 9, 30))
    for s in (2.0 ** -1060, 2.0 ** -1000, 2.0 ** 1000):
        f = N.Field.from_numpy("SVol", a * s, 1)
        want = math.fsum((a * s).reshape(-1))
        assert abs(N.nebo_sum(f) - want) <= 2.0 ** -51 * float(np.abs(a * s).sum()) + 5e-324 * a.size
    z = N.Field.from_numpy("SVol", np.zeros((12, 9, 30)), 1)
    assert (N.nebo_sum(z), N.nebo_norm(z), N.nebo_max(z), N.nebo_min(z)) == (0.0, 0.0, 0.0, 0.0)


def test_specials():
    a = np.random.default_rng(4).normal(size=(9, 10, 70))
    a[3, 4, 5] = np.nan
    a[1, 1, 1] = -np.nan
    f = N.Field.from_numpy("SVol", a, 1)
    assert math.isnan(N.nebo_sum(f)) and math.isnan(N.nebo_norm(f))
    assert N.nebo_max(f) == np.nanmax(a) and N.nebo_min(f) == np.nanmin(a)  # NaNs never win
    a[2, 2, 2], a[5, 5, 5] = np.inf, -np.inf
    f = N.Field.from_numpy("SVol", a, 1)
    assert N.nebo_max(f) == np.inf and N.nebo_min(f) == -np.inf
    f = N.Field.from_numpy("SVol", np.full((4, 4, 4), np.nan), 1)
    assert N.nebo_max(f) == -np.inf and N.nebo_min(f) == np.inf


def test_threads_and_streams():
    rng = np.random.default_rng(5)
    arrays = [rng.normal(size=(30 + i, 31, 33)) for i in range(12)]
    fields = [N.Field.from_numpy("SVol", a, 1) for a in arrays]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        for _ in range(50):
            if N.nebo_max(fields[i], s) != arrays[i].max() or \
               abs(N.nebo_sum(fields[i], s) - math.fsum(arrays[i].reshape(-1))) > 1e-13 * np.abs(arrays[i]).sum():
                bad.append(i)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(12)]  # more threads than slots
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
