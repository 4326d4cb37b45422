"""The FP64 step in three kernels (recon, flux, update) where its launch shape
changes: one-warp or 128-thread blocks, ragged last blocks, first-order
faces, gravity, and a grid whose workspace holds only part of its rows (two
bands).  Parity with the oracle, at the tolerance of the other parity tests."""
import numpy as np
import pytest

from test_gpu_parity_2d import assert_parity, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (31, 1024), (137, 139), (138, 138), (139, 139), (1025, 33)])
def test_block_shapes(gpu_available, oracle_mod, nx, ny):
    """Around the size where the blocks change from one warp to four
    (138^2 has 38640 recon items, 139^2 has 39198; the rule's limit is
    38912), the smallest grid, and long thin ones."""
    O = oracle_mod
    p = O.random_problem_2d(nx, ny, nx + ny, ("reflective", "none", "transmissive", "reflective"),
                            "monotonized_central", 6, smooth=True)
    assert_parity(p, run_gpu(p), O.load("oracle").run_2d(p))


@pytest.mark.parametrize("n", [20, 150])
@pytest.mark.parametrize("integrator", ["muscl_hancock_2d", "godunov_first_order_2d"])
def test_gravity_and_first_order(gpu_available, oracle_mod, n, integrator):
    O = oracle_mod
    p = O.rayleigh_taylor(n, n + 3, g=2, steps=10)
    p.integrator = integrator
    assert_parity(p, run_gpu(p), O.load("oracle").run_2d(p))


def test_two_bands(gpu_available, oracle_mod):
    """4200 x 2100 needs 1.13 GB of workspace, above the 1 GB it is given:
    the rows go in two bands that recompute the faces between them.  Three
    steps, bit-identical to the oracle (no two-rarefaction faces)."""
    O = oracle_mod
    p = O.random_problem_2d(4200, 2100, 1, ("periodic", "periodic", "reflective", "transmissive"),
                            "van_leer", 3, smooth=True)
    gpu, ref = run_gpu(p), O.load("oracle").run_2d(p)
    assert_parity(p, gpu, ref)
