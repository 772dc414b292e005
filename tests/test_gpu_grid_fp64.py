"""Gridded FP64 reciprocal sum against the oracle's direct sum, at sizes above the rule's line: cubic and slab
boxes, grids with and without partial blocks of cells, atoms on the box faces, and a cluster that overflows the
buckets of its cells; and the direct sums just below the line against the grid just above.

Bars: reciprocal forces 1e-12 of their norm and energies 1e-12 of their size, the bars of the direct sums: the
window leaves about 3e-14 per term (its error bound at 16 points), the sums' rounding no more."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


def _both(s, prm, gpulib, oracle):
    g, r = abi.Context(gpulib, s.copy(), prm), abi.Context(oracle, s.copy(), prm)
    a, b = g.force_get(s.copy()), r.force_get(s.copy())
    a2 = g.force_get(s.copy())  # the grid and the buckets' counts were left clear
    g.close()
    r.close()
    for o in (a, a2):
        assert np.linalg.norm(o["f"] - b["f"]) <= 1e-12 * np.linalg.norm(b["f"])
        for k in ("uewa", "ewqLL", "ewqWL"):
            assert abs(o[k] - b[k]) <= 1e-12 * (abs(b["uewa"]) + abs(b["ewqLL"]) + abs(b[k])), k


# (14, 13): 2,744 ions, 4.5e3 k: 1.2e7 products; spacing 2.8 and rcut 2: reciprocal forces alone
@pytest.mark.parametrize("n_side,kmax,shrink", [(14, 13, 1.0), (14, 16, 1.0), (18, 12, 1.0), (16, 13, 0.12)])
def test_ions(n_side, kmax, shrink, gpulib, oracle):
    s, prm = configs.ion_lattice(n_side, kmax=kmax, shuffle=True, rcut=2.0 if shrink == 1.0 else 0.1)
    n, h = s.nmove, 0.5 * s.lx
    for x in (s.x0, s.y0, s.z0):
        x[:n] *= shrink
    s.x0[0], s.y0[1], s.z0[2], s.x0[3] = -h, h, np.nextafter(-h, 0.0), -1e-18
    _both(s, prm, gpulib, oracle)


def test_slab(gpulib, oracle):
    s, prm = configs.slab_water(nwat=700, cells=7, placement="lattice", kmax=12)
    _both(s, prm, gpulib, oracle)
