"""Sums and norms with infinities, as a serial fold gives them: infinities of one sign, and squares that
leave the doubles, give that infinity; infinities of both signs and NaNs give NaN."""
import math

import numpy as np
import pytest
import torch

import spatialops_gb300 as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 5, 6), (9, 11, 300), (60, 66, 66)])
@pytest.mark.parametrize("put,total,norm", [((np.inf,), np.inf, np.inf), ((-np.inf, -np.inf), -np.inf, np.inf),
                                            ((np.inf, -np.inf), np.nan, np.inf), ((np.inf, np.nan), np.nan, np.nan),
                                            ((1e200,), None, np.inf)])
def test_infinities(shape, put, total, norm):
    a = np.random.default_rng(31).normal(size=shape)
    at = np.random.default_rng(32).permutation(a.size)[:len(put)]
    a.reshape(-1)[at] = put
    f = N.Field.from_numpy("SVol", a, 1)
    one = torch.zeros(1, dtype=torch.float64, device="cuda")
    four = torch.zeros(4, dtype=torch.float64, device="cuda")
    N.reduce_all(f, False, four)
    for op, want, k in (("sum", total, 0), ("norm", norm, 3)):
        if want is None:
            continue
        N.reduce_async(f, op, False, one)
        for got in (N._reduce(f, op, False), one.item(), four[k].item()):
            assert (math.isnan(got) if math.isnan(want) else got == want), (op, got)


def test_overflowing_sum():
    a = np.full((6, 7, 40), 1.5e308)
    for s in (1.0, -1.0):
        assert N.nebo_sum(N.Field.from_numpy("SVol", s * a, 1)) == s * np.inf
