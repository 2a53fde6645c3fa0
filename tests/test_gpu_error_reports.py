"""A CUDA error is reported by the call that met it and by no later one: reductions after an
allocation that does not fit give their values."""
import ctypes

import pytest

import spatialops_gb300 as N

pytestmark = pytest.mark.gpu


def test_reduction_after_a_failed_allocation():
    f = N.Field("SVol", (20, 20, 20), 1)
    f.tensor.fill_(1.0)
    assert N.nebo_sum(f) == 22.0 ** 3
    for _ in range(2):
        p = ctypes.c_void_p()
        assert N.lib().nebo_alloc(1 << 50, ctypes.byref(p), None) != 0 and not p.value
        assert N.nebo_sum(f) == 22.0 ** 3
