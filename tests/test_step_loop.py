"""The order of the many-step kernel: the template that the kernel runs, with
host threads as blocks.  A failing step ends every block at that step, however
far one of them lags behind, and a wait that nothing ends gives up."""
import ctypes as C

import numpy as np
import pytest

BLOCKS = 4


def run(lib, steps, slow=-1, bad=-1, bad_step=0, absent=-1, polls=20000):
    left, done, out = np.zeros(BLOCKS, np.int32), np.zeros(BLOCKS, np.int64), np.zeros(3, np.int64)
    lib.hydro_fx_step_loop_host(C.c_int(BLOCKS), C.c_int(steps), C.c_int(slow), C.c_int(bad), C.c_int(bad_step),
                                C.c_int(absent), C.c_int(polls), left.ctypes.data_as(C.POINTER(C.c_int)),
                                done.ctypes.data_as(C.POINTER(C.c_longlong)), out.ctypes.data_as(C.POINTER(C.c_longlong)))
    return left.tolist(), done.tolist(), out.tolist()


def test_all_steps(hydro_lib):
    assert run(hydro_lib, 7) == ([1] * BLOCKS, [7] * BLOCKS, [7, 0, 1])


@pytest.mark.parametrize("slow,bad", [(0, 1), (0, 3), (2, 0), (3, 1), (1, 1)])
@pytest.mark.parametrize("bad_step", [0, 1, 3])
def test_blocks_leave_at_the_failing_step(hydro_lib, slow, bad, bad_step):
    left, done, (steps, error, active) = run(hydro_lib, 6, slow=slow, bad=bad, bad_step=bad_step)
    assert left == [2] * BLOCKS and done == [bad_step] * BLOCKS
    assert (steps, error, active) == (bad_step, 1, 0)


@pytest.mark.parametrize("absent", [0, 3])
def test_a_wait_that_nothing_ends_gives_up(hydro_lib, absent):
    left, done, (steps, error, active) = run(hydro_lib, 6, absent=absent, polls=200)
    assert left == [0 if k == absent else 3 for k in range(BLOCKS)]
    assert (steps, error, active) == (0, 5, 0)        # the spin limit's code; later launches leave at once
