"""The many-step kernel where the faces take their states in one phase or in
two (35000 faces: 131^2 has 34584, 132^2 has 35112), on grids smaller than one
block of faces, and where the last block is ragged between x and y faces: every
limiter, gravity, first-order faces and all boundaries.  Parity with the oracle,
at the tolerance of the other parity tests."""
import pytest

from test_gpu_parity_2d import assert_parity, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (5, 3), (32, 31), (65, 64), (131, 131), (132, 132), (9000, 2)])
@pytest.mark.parametrize("limiter,bc", [("minmod", ("periodic",) * 4),
                                        ("van_leer", ("reflective", "transmissive", "none", "reflective")),
                                        ("monotonized_central", ("none", "none", "periodic", "periodic"))])
def test_one_and_two_phases(gpu_available, oracle_mod, nx, ny, limiter, bc):
    O = oracle_mod
    p = O.random_problem_2d(nx, ny, nx + ny, bc, limiter, 7, smooth=True)
    assert_parity(p, run_gpu(p), O.load("oracle").run_2d(p))


@pytest.mark.parametrize("n", [20, 130, 133])
@pytest.mark.parametrize("integrator", ["muscl_hancock_2d", "godunov_first_order_2d"])
def test_gravity_and_first_order(gpu_available, oracle_mod, n, integrator):
    O = oracle_mod
    p = O.rayleigh_taylor(n, n - 3, g=2, steps=9)
    p.integrator = integrator
    assert_parity(p, run_gpu(p), O.load("oracle").run_2d(p))
