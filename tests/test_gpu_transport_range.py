"""FP64 transport over the whole range of the doubles, and its rounding.  States near the largest double
step like scaled ones (the operator is linear in phi); infinities stay where the operator puts them;
the error against extended precision (at least 64 bits of significand) is that of the four-weight form
in FP64: both round each stage's state the same number of times, so the 2-norms agree within 10 %."""
import numpy as np
import pytest

import spatialops_gb300 as N
from spatialops_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _run(phi, rest, n, steps, dt, nu):
    t = N.Transport(phi, *rest, n, dt, nu, "f64")
    t.run(steps)
    return t.phi.cpu().numpy()


@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("n", [8, 33])
def test_large_states(n, steps):
    phi, u, v, w, lam, dt, nu = W.transport_inputs(n)
    rng = np.random.default_rng(41)
    phi = W.fill_periodic(rng.uniform(1.0, 2.0, phi.shape), 2)  # 27 times its differences: up to 27
    want = _run(phi, (u, v, w, lam), n, steps, dt, nu)
    got = _run(phi * 2.0 ** 1020, (u, v, w, lam), n, steps, dt, nu)
    assert np.isfinite(got).all()
    # each face: 4 products and 3 sums of values up to 54/24 * 2, k <= 0.15, 6 faces, twice a step
    assert np.abs(got * 2.0 ** -1020 - want).max() <= steps * 2 * 6 * 8 * 2.0 ** -53 * 2.0
    one = _run(np.full_like(phi, 1.5e308), (0 * u, 0 * v, 0 * w, lam), n, steps, dt, nu)
    assert np.abs(one * 2.0 ** -1000 - 1.5e308 * 2.0 ** -1000).max() <= steps * 2.0 ** -45 * 1.5e308 * 2.0 ** -1000


def test_infinity_spreads_no_further_than_the_stencil():
    n = 16
    phi, u, v, w, lam, dt, nu = W.transport_inputs(n)
    phi[2 + 8, 2 + 8, 2 + 8] = np.inf
    got = _run(phi, (u, v, w, lam), n, 1, dt, nu)[2:-2, 2:-2, 2:-2]
    d = np.abs(np.arange(n) - 8)
    reach = d[:, None, None] + d[None, :, None] + d[None, None, :]
    assert np.isfinite(got[reach > 4]).all() and not np.isfinite(got[8, 8, 8])


def _restated(phi, vel, lam, dt, nu, steps, T, weighted):
    P, V, L = phi.astype(T), [q.astype(T) for q in vel], lam.astype(T)
    dt, nu = T(dt), T(nu)

    def rhs(p):
        out = np.zeros_like(p)
        for d in range(3):
            m1, m2, p1 = np.roll(p, 1, d), np.roll(p, 2, d), np.roll(p, -1, d)
            if weighted:
                h = T(1) / T(24)
                g = ((m2 * h + m1 * (T(-27) * h)) + p * (T(27) * h)) + p1 * -h
            else:
                g = (T(27) * (p - m1) - (p1 - m2)) / T(24)
            F = nu * ((np.roll(L, 1, d) + L) * T(0.5)) * g - V[d] * np.where(V[d] > 0, m1, p)
            out = out + (np.roll(F, -1, d) - F)
        return out

    for _ in range(steps):
        one = P + dt * rhs(P)
        P = T(0.5) * P + T(0.5) * (one + dt * rhs(one))
    return P


@pytest.mark.parametrize("n,steps", [(24, 1), (24, 8), (31, 4)])
def test_error_against_extended_precision(n, steps):
    phi, u, v, w, lam, dt, nu = W.transport_inputs(n)
    c = (slice(2, -2),) * 3
    args = (phi[c], (w[c], v[c], u[c]), lam[c], dt, nu, steps)
    exact = _restated(*args, np.longdouble, False)
    err = lambda x: float(np.sqrt((((x - exact) ** 2).sum()) / (exact ** 2).sum()))  # noqa: E731
    got = _run(phi, (u, v, w, lam), n, steps, dt, nu)[c]
    assert err(got) <= 1.1 * err(_restated(*args, np.float64, True))
