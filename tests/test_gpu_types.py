"""Systems of many site types: the tables of the real-space loops in shared memory, 42 types in the mixed form and 75
in FP64, against the oracle.

Bars: FP64 forces and energies by pair type 1e-12 of their norm; mixed forces 1e-5, energies 1e-6 of the sum of
their magnitudes, as for the few-type systems."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs
from md_sim_gb300 import system as S

pytestmark = pytest.mark.gpu


def many(types, per=6):
    """`types` - 2 kinds of ions (the other two types are the empty wall's), some with vdW terms, alternating charges."""
    kinds, n = types - 2, (types - 2) * per
    side = int(np.ceil(n ** (1 / 3)))
    box = 3.2 * side
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(types)
    pos = rng.permutation(g)[:n] * 3.2 + rng.uniform(-0.2, 0.2, (n, 3)) - 0.5 * box
    names = [f"A{k}" for k in range(kinds)] + ["X1", "X2"]
    mol = [S.MolType(names[k], "atmol", per, [names[k]], [1], [0.03], [1.0 - 2.0 * (k % 2)], ns=1) for k in range(kinds)]
    crys = S.MolType("none", "crystal", 1, ["X1", "X2"], [1, 1], [1e-3, 1e-3], [0.0, 0.0], ns=0, cx=box, cy=box, cz=box, lw=box)
    pairs = {(i, j): ("LeJo", 2.5 + 0.01 * i, 0.1 + 0.01 * j) if (i + j) % 3 else ("Buck", 900.0, 0.25, 20.0 + i)
             for i in range(1, kinds + 1) for j in range(i, kinds + 1) if (i * j) % 2}
    s = S.System(S.FieldFile(mol + [crys], configs._vdw_table(names, pairs)), S.TopFile([], [], [], []), box, box, box, 1.0)
    s.x0[:n], s.y0[:n], s.z0[:n] = pos.T
    s.temper = -1.0
    return s, abi.RunParams(rcut=6.0, skin=0.5, kmax=4, alpha=0.35, variant=abi.MDG_BULK, pbc_z_list=1)


@pytest.mark.parametrize("types,precision", [(20, abi.MDG_FP64), (75, abi.MDG_FP64), (20, abi.MDG_MIXED), (42, abi.MDG_MIXED)])
def test_many_types(types, precision, gpulib, oracle):
    s, prm = many(types)
    assert s.nit == types
    g = abi.Context(gpulib, s.copy(), abi.RunParams(**{**prm.__dict__, "precision": precision}))
    r = abi.Context(oracle, s.copy(), prm)
    a, b = g.force_get(s.copy()), r.force_get(s.copy())
    g.close()
    r.close()
    force, energy = (1e-5, 1e-6) if precision == abi.MDG_MIXED else (1e-12, 1e-12)
    assert np.linalg.norm(a["f"] - b["f"]) <= force * np.linalg.norm(b["f"])
    for k in ("elj", "eqq"):
        assert np.abs(a[k] - b[k]).max() <= energy * np.abs(b[k]).sum(), k
