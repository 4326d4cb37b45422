"""The FP32 step's work items as a run plans them and the kernel decodes them:
every interior row of every strip exactly once, at one-row items, ragged last
chunks and the tallest items alike."""
import ctypes as C

import numpy as np
import pytest

STRIP = 126


def items(lib, nx, ny, g, slots):
    h = C.c_int()
    n = lib.hydro_fx_fp32_items_host(nx, ny, g, slots, C.byref(h), None, 0)
    rows = np.zeros((n, 3), np.int32)
    assert lib.hydro_fx_fp32_items_host(nx, ny, g, slots, C.byref(h), rows.ctypes.data_as(C.POINTER(C.c_int)), n) == n
    return h.value, rows


@pytest.mark.parametrize("g", [2, 3])
@pytest.mark.parametrize("slots", [0, 152, 1064])
@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 260), (64, 64), (126, 17), (127, 129), (301, 200), (130, 7), (700, 900),
                                   (1000, 4096), (2048, 2048), (8192, 8192)])
def test_every_row_once(hydro_lib, nx, ny, g, slots):
    height, rows = items(hydro_lib, nx, ny, g, slots)
    strips = (nx + STRIP - 1) // STRIP
    seen = np.zeros((strips, ny), np.int32)
    for strip, r0, r1 in rows:
        assert 0 <= strip < strips and g <= r0 < r1 <= g + ny and r1 - r0 <= height
        seen[strip, r0 - g:r1 - g] += 1
    assert np.all(seen == 1)
    assert len(rows) == strips * -(-ny // height)


def test_heights_follow_the_size(hydro_lib):
    heights = [items(hydro_lib, n, n, 2, 1064)[0] for n in (64, 512, 1024, 2048, 4096)]
    assert heights == sorted(heights) and heights[0] == 1 and heights[-1] > 12
