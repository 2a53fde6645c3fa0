"""nebo_sum keeps every element's rounding error, whatever the rows' width: on fields whose elements
cancel, the sum is the correctly rounded one within 2^-52 of itself and 2^-96 of the sum of
magnitudes (the pairs that carry sum and error hold 106 bits, and at most 2^10 of them are merged)."""
import math

import numpy as np
import pytest

import spatialops_gb300 as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interior", [False, True])
@pytest.mark.parametrize("shape", [(10, 9, 11), (20, 18, 66), (34, 40, 66), (7, 30, 255)])
def test_cancelling_sums(shape, interior):
    rng = np.random.default_rng(21)
    a = rng.normal(size=shape) * np.exp(rng.uniform(-12, 12, shape))
    flat = a.reshape(-1)
    half = flat.size // 2
    flat[half:2 * half] = -flat[:half][rng.permutation(half)] * (1 + 2.0 ** -40)  # cancels to about 2^-40
    for scale in (1.0, 2.0 ** -950, 2.0 ** 980):
        f = N.Field.from_numpy("SVol", a * scale, 1)
        r = (a[1:-1, 1:-1, 1:-1] if interior else a).reshape(-1) * scale
        want = math.fsum(r)
        got = (N.nebo_sum_interior if interior else N.nebo_sum)(f)
        assert abs(got - want) <= 2.0 ** -52 * abs(want) + 2.0 ** -96 * math.fsum(np.abs(r))


def test_norm_of_wide_ranges():
    a = np.random.default_rng(22).normal(size=(12, 20, 66)) * np.exp(np.linspace(-40, 0, 66))
    got = N.nebo_norm(N.Field.from_numpy("SVol", a, 1))
    want = math.sqrt(math.fsum(a.reshape(-1) ** 2))  # the products rounded, as there
    assert abs(got - want) <= 2.0 ** -52 * want
