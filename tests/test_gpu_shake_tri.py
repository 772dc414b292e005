"""SHAKE of three-atom, three-constraint molecules (register form) against the general form of the same
library and the oracle: the general form is reached by giving one molecule its constraints in another
order, which no molecule depends on.  Positions to the bit where only the form differs, sweep counts
equal; molecules across the periodic boundary, both stop rules, block remainders."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


def _shake(lib, s, prm, ft):
    s = s.copy()
    ctx = abi.Context(lib, s, prm)
    r = ctx.shake(s, ft)
    ctx.close()
    return np.stack([s.x0, s.y0, s.z0]), r


@pytest.mark.parametrize("nwat,clean", [(1, True), (31, True), (33, False), (96, True), (96, False)])
def test_register_form_matches_general_form_and_oracle(nwat, clean, gpulib, oracle):
    s, prm = configs.shake_water(nwat=96, cells=4, seed=11, clean=clean)
    if nwat < 96:  # the first molecules only
        t, _ = configs.shake_water(nwat=96, cells=4, seed=11, clean=clean)
        s.ncons = nwat
        s.constra, s.constrb, s.ictype = t.constra[:, :nwat].copy(), t.constrb[:, :nwat].copy(), t.ictype[:nwat].copy()
    # some molecules one box edge away from their previous positions' image, some split by the boundary
    k = np.arange(96) * 3
    for a in (0, 1, 2):
        s.x0[k[::5] + a] += s.lx
        s.y0[k[1::7] + a] -= s.ly
    s.x0[k[::9] + 1] -= s.lx
    s.xold[k[::9] + 1] -= s.lx
    ft = np.random.default_rng(3).normal(0.0, 20.0, size=(3, s.nmove))
    x, r = _shake(gpulib, s, prm, ft)
    g = s.copy()
    g.constra, g.constrb = s.constra.copy(), s.constrb.copy()
    g.constra[0, 0], g.constrb[0, 0] = s.constrb[0, 0], s.constra[0, 0]  # (1, 0): the general form for all
    y, q = _shake(gpulib, g, prm, ft)
    if clean and nwat > 1:
        np.testing.assert_array_equal(x[:, 3:], y[:, 3:])
    else:
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-9)
    assert r["sweeps"] == q["sweeps"]
    z, o = _shake(oracle, s, prm, ft)
    assert r["sweeps"] == o["sweeps"]
    np.testing.assert_allclose(x, z, rtol=0, atol=1e-9)
