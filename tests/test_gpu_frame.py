"""mdg_get_state into pinned arrays (copy kernels of 24 arrays each) and pageable ones (copies), all of them, a
part, and mixed: the same bits as a frame read through the System."""
import ctypes as C

import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["pinned", "pageable", "mixed"])
def test_frame(which, gpulib):
    torch = pytest.importorskip("torch")
    s, prm = configs.slab_electrolyte()
    c = abi.Context(gpulib, s, abi.RunParams(**{**prm.__dict__, "precision": abi.MDG_MIXED}))
    c.set_state(s)
    c.run(3)
    ref = s.copy()
    c.get_state(ref)
    keep, frame = [], abi.State()

    def take(n, k):
        pin = which == "pinned" or (which == "mixed" and k % 3)
        t = torch.zeros(max(n, 1), dtype=torch.float64)
        keep.append(t.pin_memory() if pin else t)
        a = keep[-1].numpy()[:n]
        return a, a.ctypes.data_as(abi.DP)

    got, k = [], 0
    for name in ("x0", "y0", "z0", "rsx", "rsy", "rsz"):
        a, p = take(s.ntota, k)
        setattr(frame, name, p)
        got.append((a[:s.nmove], getattr(ref, name)[:s.nmove]))
        k += 1
    for d in range(5):
        for i, (cc, ww) in enumerate(((frame.cx, frame.wx), (frame.cy, frame.wy), (frame.cz, frame.wz))):
            for dst, src in ((cc, ref.c), (ww, ref.w)):
                a, p = take(s.nrig, k)
                dst[d] = p
                got.append((a, src[d][i]))
                k += 1
        for q in range(4):
            a, p = take(s.nrig, k)
            frame.q[q][d] = p
            got.append((a, ref.q[d][q]))
            k += 1
    assert k > 48  # more than two kernels' worth
    c._check(gpulib.get_state(c.h, C.byref(frame)))
    for a, b in got:
        np.testing.assert_array_equal(a, b)
    c.close()
