"""Predictor and corrector of small systems (16 molecules per block, a component per thread) against the
oracle: molecules that fill a block, leave it short or start the next, ions beside them that do the same
with their blocks; and both sides of the line to the form with one thread per molecule.

Bars: those of the other resident FP64 comparisons (1e-9 of the box, of each derivative's largest value and of
the energies); mixed against FP64 1e-6 of the box and 2e-5 of the energies."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


def _run(lib, s, prm, steps):
    s = s.copy()
    c = abi.Context(lib, s, prm)
    c.set_state(s)
    r = c.run(steps)
    c.get_state(s)
    c.close()
    return s, r


def _close(a, ra, b, rb, pos, e, derivatives):
    for u, w in ((a.x0, b.x0), (a.y0, b.y0), (a.z0, b.z0)):
        assert np.abs(u - w).max() < pos * b.lx
    if derivatives:
        for k in range(5):
            for u, w in ((a.c[k], b.c[k]), (a.w[k], b.w[k]), (a.q[k], b.q[k])):
                assert np.abs(u - w).max() <= 10 * pos * max(np.abs(w).max(), b.lx if k == 0 and w is b.c[k] else 1e-300)
    for key in ("kp", "kw", "ke", "uconf"):
        assert abs(ra[key] - rb[key]) <= e * (abs(rb[key]) + 1.0), key


@pytest.mark.parametrize("nwat,npair,nvt", [(31, 1, False), (32, 16, False), (33, 17, True), (95, 33, True)])
def test_blocks(nwat, npair, nvt, gpulib, oracle):
    s, prm = configs.slab_electrolyte(nwat=nwat, npair=npair)
    if nvt:
        s.temper = 300.0
    b, rb = _run(oracle, s, prm, 6)
    a, ra = _run(gpulib, s, prm, 6)
    _close(a, ra, b, rb, 1e-9, 1e-9, True)


def test_mixed_partial_block(gpulib, oracle):
    s, prm = configs.bulk_water(7, "sc")  # 343 molecules: 21 blocks and 7 molecules
    b, rb = _run(oracle, s, prm, 4)
    m, rm = _run(gpulib, s, abi.RunParams(**{**prm.__dict__, "precision": abi.MDG_MIXED}), 4)
    _close(m, rm, b, rb, 1e-6, 2e-5, False)


@pytest.mark.parametrize("n_side", [22, 23])  # 10,648 and 12,167 molecules: below and above the line
def test_line(n_side, gpulib, oracle):
    s, prm = configs.bulk_water(n_side, "sc", rcut=6.0, alpha=0.45, kmax=3)
    b, rb = _run(oracle, s, prm, 2)
    a, ra = _run(gpulib, s, prm, 2)
    _close(a, ra, b, rb, 1e-9, 1e-9, True)


@pytest.mark.parametrize("fn", [lambda: configs.bulk_water(7, "sc"), lambda: configs.slab_electrolyte()])
def test_merge_blocks(fn, gpulib):
    """Site forces, centre forces and torques of a mixed force call from the merge by sites, against the FP64
    form: a last block of 23 molecules, and 24 ions beside full blocks.  Bar: the mixed forces' 1e-5 of the norm."""
    s, prm = fn()
    out = []
    for p in (abi.MDG_FP64, abi.MDG_MIXED):
        c = abi.Context(gpulib, s.copy(), abi.RunParams(**{**prm.__dict__, "precision": p}))
        out.append(c.force_get(s.copy()))
        c.close()
    a, b = out
    for key in ("f", "ft", "fc", "torque"):
        if a[key].size:
            assert np.linalg.norm(b[key] - a[key]) <= 1e-5 * np.linalg.norm(a[key]), key
