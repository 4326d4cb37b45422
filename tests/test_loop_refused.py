"""Small FP64 grids where the driver refuses the many-step kernel's cooperative
launch (a process that may use a part of the SMs): the steps are left for the
three-launch form; any other error is the run's."""
import ctypes as C

import numpy as np
import pytest

NOT_SUPPORTED, NOT_PERMITTED, TOO_LARGE = 801, 800, 720
ILLEGAL_ADDRESS, OUT_OF_RESOURCES = 700, 701


def steps(lib, k, at, code, most=10):
    out = np.zeros(3, np.int64)
    e = lib.hydro_fx_loop_steps_host(C.c_longlong(k), C.c_int(most), C.c_int(at), C.c_int(code),
                                     out.ctypes.data_as(C.POINTER(C.c_longlong)))
    return e, out.tolist()


@pytest.mark.parametrize("k", [0, 1, 10, 11, 25])
def test_granted(hydro_lib, k):
    assert steps(hydro_lib, k, -1, 0) == (0, [k, 0, 7])


@pytest.mark.parametrize("code", [TOO_LARGE, NOT_SUPPORTED, NOT_PERMITTED])
@pytest.mark.parametrize("at,done", [(0, 0), (2, 20)])
def test_refused(hydro_lib, code, at, done):
    assert steps(hydro_lib, 25, at, code) == (0, [done, 25 - done, 0])


@pytest.mark.parametrize("code", [ILLEGAL_ADDRESS, OUT_OF_RESOURCES])
def test_other_errors(hydro_lib, code):
    assert steps(hydro_lib, 25, 1, code)[0] == code
