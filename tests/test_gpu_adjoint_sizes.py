"""The reverse sweep on either side of the size up to which it takes the faces
as they come (60000 padded cells: 240 x 240 has 59536 with its ghosts) and from
which it bins them by regime (241 x 250: 62230): dot products of the gradient
with a perturbation against the tangent model's."""
import numpy as np
import pytest

import hydrofv_gb300 as h
from test_gpu_adjoint import dot, interior, smooth_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 3), (33, 7), (240, 240), (241, 250), (700, 101)])
def test_dot_product(gpu_available, nx, ny):
    """The two sums run over the same products in another order, so they agree
    to rounding of the sum of the magnitudes (400000 terms at most, a few
    hundred operations each: 1e-12)."""
    p = smooth_problem(nx, ny, ("periodic", "periodic", "reflective", "transmissive"), "monotonized_central", seed=4)
    rng = np.random.default_rng(5)
    with h.Adjoint2D(p, steps=7, checkpoint_every=3) as ad:
        ad.forward()
        seed, dw0 = rng.normal(size=p.W.shape), rng.normal(size=p.W.shape)
        grad = ad.backward(seed)
        assert ad.stats()["recompute_mismatches"] == 0
        _, dwN = ad.tangent(dw0)
        assert abs(dot(seed, dwN, p) - dot(grad, dw0, p)) <= 1e-12 * dot(abs(seed), abs(dwN), p)
        assert not grad[:, ~interior(p)].any()
