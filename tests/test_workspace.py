"""The FP64 step's workspace on a device with little room: it shrinks (more and
shorter bands), and gives way to what a session asks for after it."""
import ctypes as C

import numpy as np
import pytest

NX, NY, G = 300, 200, 2
ROW = 16 * (NX + 2 * G) * 8
FULL = (NY + 2) * ROW          # one band: all rows and one on either side
OUT_OF_MEMORY = 2              # cudaErrorMemoryAllocation


def ask(lib, room, later):
    out = np.zeros(4, np.int64)
    e = lib.hydro_fx_workspace_host(C.c_int(NX), C.c_int(NY), C.c_int(G), C.c_longlong(room), C.c_longlong(later),
                                    out.ctypes.data_as(C.POINTER(C.c_longlong)))
    return e, out.tolist()


@pytest.mark.parametrize("spare", [0, 1, 10 * ROW])
def test_room_for_both(hydro_lib, spare):
    later = 50 * ROW
    assert ask(hydro_lib, FULL + later + spare, later) == (0, [FULL, FULL, 1, NY])


@pytest.mark.parametrize("left", [3, 4, 7, 50, 101, 150, 201])
def test_the_workspace_gives_way(hydro_lib, left):
    """`left` rows' worth of room beside the later memory."""
    later = 400 * ROW
    e, (before, after, bands, rows) = ask(hydro_lib, later + left * ROW, later)
    assert e == 0 and before == FULL and rows == NY
    assert 3 * ROW <= after <= left * ROW and bands >= 2


def test_no_room_for_the_later_memory(hydro_lib):
    """The request fails and the session keeps its workspace."""
    assert ask(hydro_lib, FULL, FULL + 1) == (OUT_OF_MEMORY, [FULL, FULL, 1, NY])


def test_no_room_for_a_single_row_beside_it(hydro_lib):
    """Nothing is left to step with: an error, no bands."""
    e, (before, after, bands, rows) = ask(hydro_lib, 2 * FULL, 2 * FULL - ROW)
    assert e == OUT_OF_MEMORY and (after, bands, rows) == (0, 0, 0)
