"""The staged FP64 step's pointwise arithmetic (fused multiply-adds for sums
and products, exponent steps for scalings, integer comparisons) against the
general templates, bit for bit, on the host build: ordinary states, equal
neighbours, exact ties, and every kind of operand that has to leave the
shortcuts (zeros of both signs, subnormals, exponents near both ends,
negative densities and pressures, infinities, NaN)."""
import ctypes as C

import numpy as np
import pytest

_dp = C.POINTER(C.c_double)


def _p(a):
    return a.ctypes.data_as(_dp)


def _equal(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return (a.view(np.uint64) == b.view(np.uint64)) | nan


SPECIAL = np.array([0.0, -0.0, 5e-324, -5e-324, 2.3e-308, -2.3e-308, 4.5e-308, 1e-300, -1e-300, 1e-250, 1e-77, 1e-75,
                    1e75, 1e77, 1e250, -1e250, 1e300, -1e300, 1.7e308, np.inf, -np.inf, np.nan, 1.0, -1.0, 0.5, 2.0])


def _states(rng, n, kind):
    """n states (rho, u, v, p)."""
    w = np.empty((n, 4))
    w[:, 0] = rng.uniform(0.1, 2.0, n)
    w[:, 1:3] = rng.uniform(-1.5, 1.5, (n, 2))
    w[:, 3] = rng.uniform(0.05, 2.0, n)
    if kind == "wide":
        w[:, [0, 3]] = 10.0 ** rng.uniform(-300, 300, (n, 2))
        w[:, 1:3] = rng.choice([-1.0, 1.0], (n, 2)) * 10.0 ** rng.uniform(-320, 300, (n, 2))
    elif kind == "special":
        m = rng.random((n, 4)) < 0.4
        w[m] = rng.choice(SPECIAL, m.sum())
    elif kind == "coarse":      # few significant bits: exact ties, zeros, equal neighbours
        w = np.round(w * 4.0) / 4.0
    return np.ascontiguousarray(w)


KINDS = ["plain", "wide", "special", "coarse", "near", "strong"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("gamma", [1.4, 5.0 / 3.0])
def test_face_equals_the_general_flux(hydro_lib, kind, gamma):
    rng = np.random.default_rng(11)
    n = 40000
    base = kind if kind in ("wide", "special", "coarse") else "plain"
    L = _states(rng, n, base)
    R = _states(rng, n, base)
    if kind == "near":          # neighbouring faces of a smooth flow, many of them equal
        R = L * (1.0 + rng.choice([0.0, 1e-16, 1e-9, -1e-3], (n, 4)))
    if kind == "strong":        # collisions, rarefactions up to vacuum, pressure ratios around 2
        L[:, 1] = rng.uniform(-12, 12, n)
        R[:, 3] = L[:, 3] * rng.choice([2.0, np.nextafter(2.0, 3.0), 0.5, 1e-8, 1e5, 1.0], n)
    out, ref = np.empty((n, 5)), np.empty((n, 5))
    rc, rc_ref = np.empty(n, np.int32), np.empty(n, np.int32)
    ip = C.POINTER(C.c_int)
    hydro_lib.hydro_fx_staged_face_host(C.c_double(gamma), C.c_double(1e-6), C.c_longlong(n), _p(L), _p(R), _p(out),
                                        rc.ctypes.data_as(ip), _p(ref), rc_ref.ctypes.data_as(ip))
    assert np.array_equal(rc, rc_ref)
    good = rc == 0              # a failed face leaves no flux
    assert np.array_equal(out[:, 4], ref[:, 4])
    assert _equal(out[good], ref[good]).all()
    if kind == "strong":
        assert set(np.unique(out[:, 4])) == {0.0, 1.0, 2.0, 3.0}      # every regime


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("limiter", [1, 2, 3])
@pytest.mark.parametrize("dtA", [0.013, 1e-280])
def test_cell_equals_the_general_predictor_and_conversion(hydro_lib, kind, limiter, dtA):
    rng = np.random.default_rng(12)
    n = 30000
    base = kind if kind in ("wide", "special", "coarse") else "plain"
    wm, w0, wp = (_states(rng, n, base) for _ in range(3))
    if kind == "near":
        e = rng.choice([0.0, 2e-16, 1e-8], (n, 4))
        wm, wp = w0 * (1.0 - e), w0 * (1.0 + e * rng.choice([0.0, 0.5, 1.0, 3.0], (n, 4)))
    if kind == "strong":        # still gas beside motion that dies out through the subnormals
        w0[:, 1:3] = 0.0
        wm[:, 1:3] = 0.0
        wp[:, 1:3] = rng.choice([-1.0, 1.0], (n, 2)) * 10.0 ** rng.uniform(-324, -280, (n, 2))
    out, ref = np.empty((n, 12)), np.empty((n, 12))
    hydro_lib.hydro_fx_staged_cell_host(C.c_int(limiter), C.c_double(1.4), C.c_double(dtA), C.c_longlong(n), _p(wm),
                                        _p(w0), _p(wp), _p(out), _p(ref))
    bad = ~_equal(out, ref)
    assert not bad.any(), (np.argwhere(bad)[:3], out[bad][:3], ref[bad][:3])
