"""Sessions in a device whose memory is nearly used up: the workspace of the
FP64 step gives way to what a session keeps besides (a solver's initial state,
the adjoint's tape), and the results are those of an empty device."""
import numpy as np
import pytest

import hydrofv_gb300 as H
from hydrofv_gb300 import problems as P

pytestmark = pytest.mark.gpu

MB = 1 << 20


def session(p, steps):
    with H.Solver2D(p.nx, p.ny, p.g, (p.x_min, p.x_max, p.y_min, p.y_max), p.gamma, p.W, p.U, bc=p.bc,
                    slope_limiter=p.slope_limiter, cfl=p.cfl) as s:
        s.advance(steps)
        s.restart()
        s.advance(steps)
        return s.download()


def gradient(p, steps):
    with H.Adjoint2D(p, steps, steps) as a:
        a.forward()
        seed = np.ones((4, p.ny + 2 * p.g, p.nx + 2 * p.g))
        g = a.backward(seed)
        return g, a.stats()["device_bytes"]


class Ballast:
    """All device memory but `left` bytes, taken."""

    def __init__(self, torch, left):
        self.torch = torch
        assert H.library().hydro_gpu_trim_device_memory(0) == 0
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        assert free > left
        self.mem = torch.empty(free - left, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.mem = None
        self.torch.cuda.empty_cache()


def test_session(gpu_available):
    torch = pytest.importorskip("torch")
    p = P.shear_layer(2048)
    want = session(p, 3)
    field = (p.nx + 2 * p.g) * (p.ny + 2 * p.g) * 8
    # 22 fields of state and 8 of the initial state; less than the workspace's 16 fields are left
    with Ballast(torch, 30 * field + 400 * MB):
        got = session(p, 3)
    for x, y in zip(want, got):
        assert np.array_equal(x, y, equal_nan=True)      # (NaN in ghost corners)


def test_adjoint(gpu_available):
    torch = pytest.importorskip("torch")
    p = P.shear_layer(1024)
    want, used = gradient(p, 2)
    field = (p.nx + 2 * p.g) * (p.ny + 2 * p.g) * 8
    with Ballast(torch, used - 10 * field + 8 * MB):
        got, _ = gradient(p, 2)
    assert np.array_equal(want, got)
