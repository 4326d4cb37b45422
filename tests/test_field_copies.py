"""States copied into and out of a System's fields, on either side of the size
from which the copies run in several threads (2 million numbers: 500000 cells
out, 250000 in)."""
import numpy as np
import pytest

import hydrofv_gb300 as H


@pytest.mark.parametrize("nx,ny", [(3, 2), (495, 495), (497, 499), (703, 703), (705, 707), (1500, 401)])
def test_fill_and_copies(nx, ny):
    h = H._SystemHandle(H.library(), "cartesian_2d", nx, ny, 2, (0.0, 1.0, 0.0, 1.0), 1.4)
    rng = np.random.default_rng(nx)
    W, U = rng.normal(size=(2, 4) + h.shape)
    h.fill(H.W2, [*W[:2], W[2].astype(np.float32), W[3, ::-1]], H.U2, U)
    W[2] = W[2].astype(np.float32)
    W[3] = W[3, ::-1].copy()
    a, b = h.copies(H.W2), h.copies(H.U2)
    h.close()
    assert np.array_equal(a, W) and np.array_equal(b, U)
    assert a.flags.owndata and a.flags.c_contiguous
