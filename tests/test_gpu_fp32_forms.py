"""The FP32 step's short quotients, roots and slopes, and the faces and cells
made of them, against the general forms on the device: bit for bit, up to the
bounds between which the short forms are taken and beyond them."""
import numpy as np
import pytest

import hydrofv_gb300 as H

pytestmark = pytest.mark.gpu

N = 200000


def same(x, y):
    return (x.view(np.uint32) == y.view(np.uint32)) | (np.isnan(x) & np.isnan(y))


def log_uniform(rng, lo, hi, shape):
    return 10.0 ** rng.uniform(np.log10(lo), np.log10(hi), shape)


def states(rng, lo, hi, speed):
    """n states (rho, u, v, p) whose density and pressure lie between lo and hi."""
    w = np.empty((N, 4), np.float32)
    w[:, 0] = log_uniform(rng, lo, hi, N)
    w[:, 3] = log_uniform(rng, lo, hi, N)
    w[:, 1:3] = rng.choice([-1.0, 1.0], (N, 2)) * log_uniform(rng, 1e-6 * speed, speed, (N, 2))
    return w


def test_quotient_and_root(gpu_available):
    """Within 2 ulp (quotient) and one part in 2^-22 (root) of the exact value."""
    rng = np.random.default_rng(1)
    a = (rng.choice([-1.0, 1.0], N) * 2.0 ** rng.uniform(-60, 60, N)).astype(np.float32)
    b = (rng.choice([-1.0, 1.0], N) * 2.0 ** rng.uniform(-60, 60, N)).astype(np.float32)
    q, _ = H.gpu_fp32_eval("quotient", a, b)
    exact = a.astype(np.float64) / b.astype(np.float64)
    assert np.all(np.abs(q - exact) <= 2.0 * np.spacing(np.abs(exact).astype(np.float32)))
    r, _ = H.gpu_fp32_eval("root", np.abs(a))
    assert np.all(np.abs(r - np.sqrt(np.abs(a).astype(np.float64))) <= 2.0 ** -22 * r)


@pytest.mark.parametrize("gamma", [1.1, 1.4, 5.0 / 3.0])
@pytest.mark.parametrize("lo,hi,speed,near", [(0.1, 10.0, 1.0, True), (1e-3, 1e3, 30.0, False), (1e-12, 1e8, 1e8, False),
                                              (1e-14, 1e-10, 1e-3, False), (1e6, 1e10, 1e9, False)])
def test_faces(gpu_available, gamma, lo, hi, speed, near):
    rng = np.random.default_rng(2)
    L, R = states(rng, lo, hi, speed), states(rng, lo, hi, speed)
    if near:                       # a smooth flow: neighbours a little apart, some equal
        R = (L * (1.0 + rng.choice([0.0, 1e-6, 1e-3, 0.1], (N, 1)) * rng.standard_normal((N, 4)))).astype(np.float32)
    x, y = H.gpu_fp32_eval("flux", L, R, gamma=gamma)
    bad = ~same(x, y)
    assert not bad.any(), (bad.any(axis=1).sum(), L[bad.any(axis=1)][:3], R[bad.any(axis=1)][:3], x[bad.any(axis=1)][:3],
                           y[bad.any(axis=1)][:3])


@pytest.mark.parametrize("vol", [1e-6, 1.0, 1e11])
@pytest.mark.parametrize("lo,hi", [(1e-3, 1e3), (1e-27, 1e-20), (1e9, 1e14)])
def test_cells(gpu_available, lo, hi, vol):
    rng = np.random.default_rng(3)
    U = np.empty((N, 4), np.float32)
    U[:, 0] = log_uniform(rng, lo, hi, N)
    u = rng.choice([0.0, 1e-6, 1.0, 10.0], (N, 2)) * rng.standard_normal((N, 2))
    U[:, 1:3] = U[:, :1] * u
    U[:, 3] = U[:, 0] * (0.5 * (u ** 2).sum(axis=1) + log_uniform(rng, 1e-8, 1e2, N) * rng.choice([1.0, 1.0, -1.0, 0.0], N))
    x, y = H.gpu_fp32_eval("primitive", U, vol=vol)
    assert same(x, y).all()


@pytest.mark.parametrize("limiter", ["minmod", "van_leer", "mc"])
def test_slopes(gpu_available, limiter):
    rng = np.random.default_rng(4)
    a, b = (rng.choice([-1.0, 1.0], N) * log_uniform(rng, 1e-40, 1e20, N) for _ in range(2))
    b = np.where(rng.random(N) < 0.5, a * rng.choice([-3.0, -1.0, 0.3, 0.5, 1.0, 2.0, 3.0], N), b)
    special = [0.0, -0.0, 1.0, -1.0, 1e-45, -1e-45, 3e38, -3e38]
    a[:64], b[:64] = (x.ravel() for x in np.meshgrid(special, special))
    x, y = H.gpu_fp32_eval("slope_" + limiter, a, b)
    bad = ~same(x, y)
    assert not bad.any(), (a[bad][:5], b[bad][:5], x[bad][:5], y[bad][:5])
