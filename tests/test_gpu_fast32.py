"""FP32 faces and cells in the short quotients, roots and powers against the
same ones in the compiler's general forms.  Density, pressure and the conserved
values times a power of two leave every other number of the scheme as it is, and put the
states beyond the bounds (1e8) up to which the short forms are taken: 2^26
leaves some faces on either side, 2^60 takes all faces and cells to the
general forms."""
import numpy as np
import pytest

import hydrofv_gb300 as H
from hydrofv_gb300 import problems as P

pytestmark = pytest.mark.gpu

STEPS = 5
# Powers are the only numbers that do not scale exactly: p^(1/12) (gamma = 1.2)
# and its 12th power, each to 2 ulp, are within 32 ulp of the star pressure
# (2^-19).  A cell moves by less than the largest value of its field in a step.
TOL = STEPS * 2.0 ** -19


def advance(p, limiter, integrator, scale):
    W, U = p.W.copy(), p.U.copy()
    W[[0, 3]] *= scale
    U *= scale
    r = H.run_2d(p.nx, p.ny, p.g, (p.x_min, p.x_max, p.y_min, p.y_max), p.gamma, W, U, bc=p.bc,
                 slope_limiter=limiter, integrator=integrator, cfl=p.cfl, tf=p.tf, max_steps=STEPS,
                 options=H.default_options(precision=H.PRECISION_FP32))
    assert r.code == 0 and r.num_steps == STEPS, r.message
    W, U = r.W.copy(), r.U.copy()
    W[[0, 3]] /= scale
    return r, W, U / scale


@pytest.mark.parametrize("log2_scale", [26, 60])
@pytest.mark.parametrize("limiter,integrator", [("minmod", "muscl_hancock_2d"), ("van_leer", "muscl_hancock_2d"),
                                                ("monotonized_central", "muscl_hancock_2d"),
                                                ("minmod", "godunov_first_order_2d")])
def test_short_and_general_forms(gpu_available, limiter, integrator, log2_scale):
    p = P.random_problem_2d(67, 41, 5, ("periodic", "periodic", "reflective", "transmissive"), limiter, STEPS,
                            smooth=False)
    a, Wa, Ua = advance(p, limiter, integrator, 1.0)
    b, Wb, Ub = advance(p, limiter, integrator, 2.0 ** log2_scale)
    assert abs(a.t - b.t) <= TOL * a.t
    for x, y in ((Wa, Wb), (Ua, Ub)):
        assert np.all(np.abs(x - y).max(axis=(1, 2)) <= TOL * np.abs(x).max(axis=(1, 2)))
