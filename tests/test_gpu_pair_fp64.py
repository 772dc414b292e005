"""FP64 pair and wall loops against the oracle: head counts on both sides of each split of the lists,
site pairs below, inside and above the range of the function table, partner queues of every length, and a
film so thin that every head has partners in both walls.

Bars: forces 1e-12 of their norm and energies 1e-12 of the terms' magnitudes, as in the other
comparisons of the two FP64 forms; wall reactions (sums of the forces) 1e-11 of the largest."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


def _both(s, prm, gpulib, oracle):
    g, r = abi.Context(gpulib, s.copy(), prm), abi.Context(oracle, s.copy(), prm)
    a, b = g.force_get(s.copy()), r.force_get(s.copy())
    g.close()
    r.close()
    assert np.isfinite(b["f"]).all() and np.linalg.norm(b["f"]) > 0.0
    assert np.linalg.norm(a["f"] - b["f"]) <= 1e-12 * np.linalg.norm(b["f"])
    for k in ("elj", "eqq"):
        assert np.abs(a[k] - b[k]).max() <= 1e-12 * (np.abs(b["elj"]).sum() + np.abs(b["eqq"]).sum())
    return a, b


# 1,000, 1,728 and 2,744 heads: lists in four parts, two and one; then (alpha r)^2 from 0.04, and to 92
@pytest.mark.parametrize("n_side,alpha,shrink", [(4, 0.35, 1.0), (10, 0.35, 1.0), (12, 0.35, 1.0), (14, 0.35, 1.0),
                                                 (6, 0.35, 0.2), (6, 1.6, 1.0)])
def test_ions(n_side, alpha, shrink, gpulib, oracle):
    s, prm = configs.ion_lattice(n_side, spacing=2.8 if n_side > 4 else 4.2, rcut=6.0, alpha=alpha, shuffle=True)
    for x in (s.x0, s.y0, s.z0):
        x[:s.nmove] *= shrink
    _both(s, prm, gpulib, oracle)


@pytest.mark.parametrize("nwat,cells", [(33, 6), (150, 6), (1040, 6)])
def test_walls_on_both_sides(nwat, cells, gpulib, oracle):
    s, prm = configs.slab_water(nwat=nwat, cells=cells, placement="lattice", kmax=4)
    a, b = _both(s, prm, gpulib, oracle)
    assert np.abs(b["fws"]).max() > 0.0
    assert np.abs(a["fws"] - b["fws"]).max() <= 1e-11 * np.abs(b["fws"]).max()
