"""FP64 Widom insertion by points (all positions' sites in one reciprocal sum) against the oracle: counts of
insertions around those that fill a block of points, one and twenty orientations, charged walls near
and far; and the limit of sites around a probe.

Bar: pave to 1e-9 of its largest bin, as in the other comparison of the two (exp(-u/kT) of energies that agree
to about 1e-12 of their terms); counts and generator state exact."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu

SEED0 = 14135621772.0


@pytest.mark.parametrize("nins,ilmid,kmax", [(1, 8, 6), (2, 0, 6), (31, 8, 3), (70, 0, 9), (300, 4, 6)])
def test_counts(nins, ilmid, kmax, gpulib, oracle):
    s, prm = configs.slab_water(nwat=96, cells=6, placement="lattice", kmax=kmax)
    out = []
    for lib in (gpulib, oracle):
        c = abi.Context(lib, s.copy(), prm)
        c.force_get(s.copy())
        out.append(c.widom(nins, 1.0, 4.0, 8, ilmid, SEED0, flags=abi.MDG_WIDOM_SKIP_OVERLAP | abi.MDG_WIDOM_EW3DC))
        c.close()
    a, b = out
    assert a["done"] == b["done"] == nins and a["seed"] == b["seed"]
    np.testing.assert_array_equal(a["inave"], b["inave"])
    assert np.abs(a["pave"] - b["pave"]).max() <= 1e-9 * max(b["pave"].max(), 1e-300), (a["pave"], b["pave"])


def test_too_many_sites_around_the_probe(gpulib):
    s, prm = configs.slab_water(nwat=2048, cells=10, placement="lattice", kmax=3, rcut=20.0)
    c = abi.Context(gpulib, s.copy(), prm)
    c.force_get(s.copy())
    with pytest.raises(Exception, match="more than 1024 sites"):
        c.widom(200, 1.0, 3.0, 8, 8, SEED0, flags=abi.MDG_WIDOM_SKIP_OVERLAP)
    c.close()


@pytest.mark.parametrize("nins,seed", [(512, SEED0), (513, SEED0), (1030, 67099546.0), (600, 12345.678), (300, 3.0e9 + 0.5)])
def test_chunks_and_seeds(nins, seed, gpulib, oracle):
    """Positions drawn in chunks, from integer states (drawn ahead) and others: the generator's state and the
    counts are the oracle's to the bit."""
    s, prm = configs.slab_water(nwat=64, cells=6, placement="lattice", kmax=3)
    out = []
    for lib in (gpulib, oracle):
        c = abi.Context(lib, s.copy(), prm)
        c.force_get(s.copy())
        out.append(c.widom(nins, 1.0, 2.0, 5, 4, seed, flags=abi.MDG_WIDOM_SKIP_OVERLAP))
        c.close()
    a, b = out
    assert a["done"] == b["done"] == nins and a["seed"] == b["seed"]
    np.testing.assert_array_equal(a["inave"], b["inave"])
    assert np.abs(a["pave"] - b["pave"]).max() <= 1e-9 * max(b["pave"].max(), 1e-300)
