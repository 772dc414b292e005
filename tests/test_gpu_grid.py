"""Gridded reciprocal sum of the mixed form (recip_nu.cu) against the FP64 form of the library, at the
sizes where it can go wrong: grids that the blocks of 8 cells do not divide, many atoms per block,
blocks whose bucket overflows, static walls, tall boxes with few atoms, replica batches.

Bars: forces 1e-5 (the metric's), the reciprocal energy 2e-6: the window and FP32 leave about 1e-6 in
the forces and 2e-7 in S(k), and an energy is quadratic in S(k)."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu

FORCE_RTOL, ENERGY_RTOL = 1e-5, 2e-6


def _ions(n_side, kmax, squeeze=1.0):
    """Point ions, charges dealt at random, no pair inside the cutoff; squeeze < 1 gathers them in a
    corner of the box."""
    s, prm = configs.ion_lattice(n_side, spacing=2.8, rcut=0.3, alpha=0.35, kmax=kmax, shuffle=True)
    for a in (s.x0, s.y0, s.z0):
        a[:s.nmove] *= squeeze
    return s, prm


CASES = {
    "blocks divide": lambda: _ions(26, 14),                   # M = 64, 17,576 atoms
    "ragged blocks": lambda: _ions(28, 13),                   # M = 60
    "many atoms per block": lambda: _ions(42, 8),             # M = 40, 593 atoms per block
    "full buckets": lambda: _ions(26, 14, squeeze=0.25),      # 64 times the density in one corner
    "walls": lambda: configs.slab_water(3600, 13, kmax=13, placement="lattice"),
    "tall box": lambda: configs.slab_water(64, 6, kmax=6, lz=6 * 4.21 * 5.6, placement="lattice"),  # knmax 34
}


@pytest.mark.parametrize("name", list(CASES))
def test_grid_sum_vs_fp64(name, gpulib):
    s, prm = CASES[name]()
    out = {}
    for p in (abi.MDG_FP64, abi.MDG_MIXED):
        ctx = abi.Context(gpulib, s.copy(), abi.RunParams(**{**prm.__dict__, "precision": p}))
        out[p] = [ctx.force_get(s.copy()) for _ in range(2)]  # the second: buckets and grid left clean
        ctx.close()
    a = out[abi.MDG_FP64][0]
    for b in out[abi.MDG_MIXED]:
        assert np.linalg.norm(b["f"] - a["f"]) <= FORCE_RTOL * np.linalg.norm(a["f"])
        assert abs(b["uewa"] - a["uewa"]) <= ENERGY_RTOL * abs(a["uewa"])
        assert abs(b["ewqLL"] - a["ewqLL"]) <= ENERGY_RTOL * abs(a["ewqLL"])


def test_grid_sum_in_a_batch(gpulib):
    """A replica with the gridded sum beside one with the tensor-core sum, against each stepped alone."""
    def build():
        sy = [CASES["tall box"](), configs.slab_water(256, 6, seed=40, kmax=6, placement="lattice")]
        for _, p in sy:
            p.precision = abi.MDG_MIXED
        ctxs = [abi.Context(gpulib, s, p) for s, p in sy]
        for c in ctxs:
            c.set_state(c.sys)
        return ctxs

    together, alone = build(), build()
    batch = abi.Batch(gpulib, together)
    reps = batch.run(8)
    for c, d, r in zip(together, alone, reps):
        one = d.run(8)
        c.get_state()
        d.get_state()
        # FP32 sums in another order (as for the tensor-core replicas of the batch tests)
        assert np.abs(c.sys.x0 - d.sys.x0).max() < 1e-7 * c.sys.lx
        assert abs(r["uconf"] - one["uconf"]) <= 1e-5 * abs(one["uconf"])
    batch.close()
