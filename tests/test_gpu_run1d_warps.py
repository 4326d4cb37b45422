"""The 1D run where its warps are dealt out (one or none per CTA, the last warp
ragged, more cells than threads), where whole warps meet equal states (gas at
rest, moving gas, -0 velocities, a pressure below the tolerance), and the
geometry source taken with the update on every kind of boundary.  Parity with
the oracle, at the tolerance of the other 1D tests."""
import numpy as np
import pytest

from hydrofv_gb300.problems import random_problem_1d, sedov_1d
from test_gpu_parity_1d_godunov import REL_L1_TOL, rel_l1_1d, run1

pytestmark = pytest.mark.gpu


def assert_parity(O, p):
    ref, r = O.load("oracle").run_1d(p), run1(p)
    assert (r.code == 0) == (ref.rc == 0), (r.message, ref.message)
    if ref.rc != 0:             # a state that the scheme refuses (Sedov without a left boundary)
        return
    assert r.num_steps == ref.num_steps and abs(r.t - ref.t) <= 1e-13 * ref.t
    assert np.all(rel_l1_1d(r.U, ref.U, p.g) <= REL_L1_TOL)
    assert np.all(np.abs(r.W - ref.W) <= 1e-11 * np.abs(ref.W).max(axis=1, keepdims=True))


@pytest.mark.parametrize("n", [27, 508, 1023, 4092, 4100, 9001])
@pytest.mark.parametrize("solver", ["riemann_solver_exact", "riemann_solver_hllc"])
@pytest.mark.parametrize("u", [0.0, -0.0, 0.7])
def test_equal_states_beside_a_wave(gpu_available, oracle_mod, n, solver, u):
    p = random_problem_1d(n, 3, ("transmissive", "reflective"), "godunov_first_order_1d", solver, "minmod", steps=6)
    W, x = p.W, np.arange(p.W.shape[1])
    for lo, hi, rho, pr in ((0.0, 0.3, 1.0, 1.0), (0.5, 0.9, 0.3, 1e-7)):
        m = (x >= lo * n) & (x < hi * n)
        W[0][m], W[1][m], W[2][m] = rho, u, pr
    vol = (p.x_max - p.x_min) / W.shape[1]
    p.U[0] = W[0] * vol
    p.U[1] = p.U[0] * W[1]
    p.U[2] = vol * (0.5 * W[0] * W[1] * W[1] + W[2] / (p.gamma - 1.0))
    assert_parity(oracle_mod, p)


@pytest.mark.parametrize("coord", ["cylindrical_1d", "spherical_1d"])
@pytest.mark.parametrize("bc", [("reflective", "transmissive"), ("none", "none"), ("reflective", "reflective")])
@pytest.mark.parametrize("integ,lim", [("godunov_first_order_1d", "minmod"), ("muscl_hancock_1d", "van_leer"),
                                       ("muscl_hancock_1d", "monotonized_central")])
def test_source_with_the_update(gpu_available, oracle_mod, coord, bc, integ, lim):
    p = sedov_1d(300, coord_sys=coord, steps=40)
    p.integrator, p.riemann_solver, p.slope_limiter, p.bc = integ, "riemann_solver_hllc", lim, bc
    assert_parity(oracle_mod, p)
