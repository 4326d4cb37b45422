"""The FP64 step in three stages (recon, flux, update) where its launch shape
changes: many steps in one cooperative launch or three launches a step, ragged
last blocks, first-order faces, gravity, stopping times and snapshots inside a
launch, and a grid whose workspace holds only part of its rows (two bands).  Parity with the oracle, at the tolerance of the other parity tests."""
import numpy as np
import pytest

from test_gpu_parity_2d import assert_parity, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (31, 1024), (137, 139), (315, 315), (316, 316), (1025, 33)])
def test_block_shapes(gpu_available, oracle_mod, nx, ny):
    """The smallest grid, long thin ones, and around the largest that steps in
    the many-step kernel (315^2 has 199710 recon items, 316^2 has 200976; the
    rule's limit is 200000)."""
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


@pytest.mark.parametrize("n", [40, 330])
def test_stopping_time(gpu_available, oracle_mod, n):
    """A run to tf (the last dt is clipped, the steps past it are not taken)
    in either form, and a session whose stopping time moves between calls."""
    import hydrofv_gb300 as H
    O = oracle_mod
    p = O.random_problem_2d(n, n, 3, ("periodic",) * 4, "minmod", -1, smooth=True)
    p.tf = 0.012
    ref = O.load("oracle").run_2d(p)
    assert_parity(p, run_gpu(p), ref)
    with H.Solver2D(p.nx, p.ny, p.g, (p.x_min, p.x_max, p.y_min, p.y_max), p.gamma, p.W, p.U, bc=p.bc,
                    slope_limiter=p.slope_limiter, cfl=p.cfl) as s:
        st, _ = s.advance(3)
        assert st.num_steps == 3
        st, _ = s.advance(1000, tf=p.tf)
        assert st.num_steps == ref.num_steps and st.t == ref.t and st.dt == ref.dt
        W, U = s.download()
    assert np.all(O.rel_l1(U, ref.U, p.g) <= 1e-12)


def test_two_bands(gpu_available, oracle_mod):
    """4200 x 2100 needs 1.13 GB of workspace, above the 1 GB it is given:
    the rows go in two bands that recompute the faces between them.  Three
    steps, bit-identical to the oracle (no two-rarefaction faces)."""
    O = oracle_mod
    p = O.random_problem_2d(4200, 2100, 1, ("periodic", "periodic", "reflective", "transmissive"),
                            "van_leer", 3, smooth=True)
    gpu, ref = run_gpu(p), O.load("oracle").run_2d(p)
    assert_parity(p, gpu, ref)


def _batch_equals_single(probs, steps):
    import hydrofv_gb300 as H
    with H.Batch2D(probs) as b:
        st, _ = b.advance(steps)
        outs = b.download()
    for p, (W, U), s in zip(probs, outs, st):
        r = run_gpu(p)
        assert r.code == 0 and s == (r.num_steps, r.t, r.dt)
        assert np.array_equal(U, r.U, equal_nan=True) and np.array_equal(W, r.W, equal_nan=True)


@pytest.mark.parametrize("integrator", ["muscl_hancock_2d", "godunov_first_order_2d"])
def test_batch_equals_single_grids(gpu_available, oracle_mod, integrator):
    """Instances of one to many blocks in the batch's launches against the
    single grids (the many-step kernel and the three launches)."""
    O = oracle_mod
    probs = [O.random_problem_2d(nx, ny, 7 + nx, ("reflective", "transmissive", "none", "reflective"), "van_leer", 9,
                                 smooth=True, integrator=integrator) for nx, ny in [(2, 3), (9, 11), (400, 300), (65, 130)]]
    for p in probs:
        p.cfl = 0.5
    _batch_equals_single(probs, 9)


def test_batch_groups(gpu_available, oracle_mod):
    """Three instances of 0.44 GB of workspace each: two share the 1 GB, the
    third is stepped by launches of its own."""
    O = oracle_mod
    probs = [O.random_problem_2d(2000, 1700, k, ("periodic",) * 4, "minmod", 3, smooth=True) for k in range(3)]
    _batch_equals_single(probs, 3)
