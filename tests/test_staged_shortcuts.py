"""The staged FP64 step's integer differences, sums and slopes and its test for
two rarefactions against the general templates, bit for bit, on the host build,
where they could go wrong: neighbours on either side of a power of two, of
either sign, a few units of the last place apart, at the ends of the exponent
range, gas at rest; and pairs of states around the velocity difference at which
the star pressure reaches the smaller pressure."""
import ctypes as C

import numpy as np
import pytest

from test_staged_math import _equal, _p


def _face(lib, gamma, tol, L, R):
    n = len(L)
    out, ref = np.empty((n, 5)), np.empty((n, 5))
    rc, rc_ref = np.empty(n, np.int32), np.empty(n, np.int32)
    ip = C.POINTER(C.c_int)
    lib.hydro_fx_staged_face_host(C.c_double(gamma), C.c_double(tol), C.c_longlong(n), _p(L), _p(R), _p(out),
                                  rc.ctypes.data_as(ip), _p(ref), rc_ref.ctypes.data_as(ip))
    assert np.array_equal(rc, rc_ref)
    assert _equal(out[rc == 0], ref[rc == 0]).all()
    return ref[:, 4]


@pytest.mark.parametrize("gamma", [1.00003, 1.01, 1.4, 5.0 / 3.0, 3.0])
@pytest.mark.parametrize("tol", [1e-6, 0.3])
def test_around_the_edge_of_two_rarefactions(hydro_lib, gamma, tol):
    rng = np.random.default_rng(3)
    n = 40000
    L, R = np.empty((n, 4)), np.empty((n, 4))
    for w in (L, R):
        w[:, 0] = rng.uniform(0.1, 2.0, n)
        w[:, 1:3] = rng.uniform(-1.0, 1.0, (n, 2))
        w[:, 3] = rng.uniform(0.2, 2.0, n)
    R[:, 3] = L[:, 3] * (1.0 + rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-16, -0.2, n))
    a = np.where(L[:, 3] > R[:, 3], np.sqrt(gamma * L[:, 3] / L[:, 0]), np.sqrt(gamma * R[:, 3] / R[:, 0]))
    lo, up = np.minimum(L[:, 3], R[:, 3]), np.maximum(L[:, 3], R[:, 3])
    z = (gamma - 1.0) / (2.0 * gamma)
    exact = 2.0 * a * (1.0 - (lo / up) ** z) / (gamma - 1.0)     # p* = min(p_L, p_R)
    bound = a * (up - lo) / (gamma * lo)                         # the test's
    step = rng.choice([0.0, 1e-16, 1e-13, 1e-10, 1e-9, 3e-9, 1e-6, 1e-2], n) * rng.choice([-1.0, 1.0], n)
    R[:, 1] = L[:, 1] + np.where(rng.random(n) < 0.5, exact, bound) * (1.0 + step) + np.where(rng.random(n) < 0.3, step, 0.0)
    regimes = _face(hydro_lib, gamma, tol, L, R)
    assert (regimes == 2.0).sum() > n // 10


@pytest.mark.parametrize("scale", [2.0 ** -249, 2.0 ** -240, 1.0, 2.0 ** 241, 2.0 ** 249])
@pytest.mark.parametrize("limiter", [1, 2, 3])
def test_slopes_of_close_neighbours(hydro_lib, limiter, scale):
    rng = np.random.default_rng(limiter)
    n = 60000
    w0 = rng.choice([1.0, 2.0, 0.5, 1.5, 1.0 - 2.0 ** -53, 511.0, 1.0 / 512.0], (n, 4))

    def near():
        m = rng.integers(0, 6, (n, 4))
        ulp = np.spacing(w0)
        v = np.choose(m, [w0, w0 + rng.integers(-3, 4, (n, 4)) * ulp, w0 * (1.0 + rng.uniform(-0.6, 1.2, (n, 4))),
                          w0 * 2.0 ** rng.integers(-11, 12, (n, 4)), w0 * rng.uniform(0.001, 900.0, (n, 4)),
                          w0 * (1.0 + 1e-9 * rng.standard_normal((n, 4)))])
        return v
    wm, wp = near(), near()
    flip = rng.random((n, 4)) < 0.1
    flip[:, [0, 3]] = False
    sign = np.where(rng.random((n, 4)) < 0.5, -1.0, 1.0)
    sign[:, [0, 3]] = 1.0
    w0, wm, wp = (np.ascontiguousarray(x * sign * scale) for x in (w0, np.where(flip, -wm, wm), wp))
    rest = rng.random(n) < 0.2                                    # gas at rest, zeros of either sign
    for x in (w0, wm, wp):
        x[np.ix_(rest, [1, 2])] = rng.choice([0.0, -0.0], (rest.sum(), 2))
    still = rng.random(n) < 0.2
    wm[still], wp[still] = w0[still], w0[still]
    out, ref = np.empty((n, 12)), np.empty((n, 12))
    hydro_lib.hydro_fx_staged_cell_host(C.c_int(limiter), C.c_double(1.4), C.c_double(0.01), C.c_longlong(n), _p(wm),
                                        _p(w0), _p(wp), _p(out), _p(ref))
    bad = ~_equal(out, ref)
    assert not bad.any(), (np.argwhere(bad)[:3], out[bad][:3], ref[bad][:3])
