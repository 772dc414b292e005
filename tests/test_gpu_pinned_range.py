"""Host arrays that begin in a range given to mdg_pin_host and end beyond it."""
import ctypes as C

import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("end", [4096, 4096 + 8 * 37, 4096 + 8 * 37 + 4, 4096 + 4])
def test_arrays_across_the_end_of_a_pinned_range(end, gpulib):
    """Frames and force calls on arrays that begin in a range of mdg_pin_host and end beyond it: the same numbers."""
    s, prm = configs.slab_water(400, 6, kmax=6, placement="lattice")
    c = abi.Context(gpulib, s, prm)
    c.set_state(s)
    c.run(3)
    ref = s.copy()
    c.get_state(ref)
    raw = np.zeros(4 * 4096 // 8 + 8 * s.ntota)
    first = (-raw.ctypes.data) % 4096 // 8  # a page boundary
    page = raw[first:]
    assert gpulib.pin_host(page.ctypes.data, end) == 0
    x = page[4096 // 8 - 20:][:s.ntota]  # 20 words before the boundary, most of it after the range
    frame = abi.State()
    frame.x0 = x.ctypes.data_as(abi.DP)
    c._check(gpulib.get_state(c.h, C.byref(frame)))
    np.testing.assert_array_equal(x[:s.nmove], ref.x0[:s.nmove])
    want = c.force_get(ref.copy())
    moved = ref.copy()
    x[:] = ref.x0
    moved.x0 = x
    got = c.force_get(moved)
    assert np.linalg.norm(got["f"] - want["f"]) <= 1e-12 * np.linalg.norm(want["f"])
    assert gpulib.unpin_host(page.ctypes.data) == 0
    c.close()
