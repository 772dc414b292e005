"""Mixed pair loop with partner queues against the FP64 form: a cluster of ions in which the half lists
have every length from 0 up, so that the queue of 32 is left empty, partly filled, just filled and
refilled, with every pair inside the cutoff or a part of them; both site types as heads and partners.

Bars: forces 1e-5 of their norm (the metric's); energies 1e-6 of the sum of their terms' magnitudes: FP32
terms with compensated sums, and an approximation of erfc to 1.5e-7 on both sides."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_side,rcut", [(2, 6.0), (4, 6.0), (6, 6.0), (6, 2.0)])
def test_queue_lengths_vs_fp64(n_side, rcut, gpulib):
    s, prm = configs.ion_lattice(n_side, spacing=16.8 / n_side, rcut=rcut, shuffle=True)
    n = s.nmove
    for a in (s.x0, s.y0, s.z0):
        a[:n] *= 0.2  # all ions within 5.9 A of each other
    out = {}
    for p in (abi.MDG_FP64, abi.MDG_MIXED):
        ctx = abi.Context(gpulib, s.copy(), abi.RunParams(**{**prm.__dict__, "precision": p}))
        out[p] = ctx.force_get(s.copy())
        (i, j), _ = ctx.get_lists()
        assert len(i) == len(set(zip(i.tolist(), j.tolist()))) and (rcut < 6.0 or len(i) == n * (n - 1) // 2)
        ctx.close()
    a, b = out[abi.MDG_FP64], out[abi.MDG_MIXED]
    assert np.linalg.norm(b["f"] - a["f"]) <= 1e-5 * np.linalg.norm(a["f"])
    assert np.abs(b["eqq"] - a["eqq"]).max() <= 1e-6 * np.abs(a["eqq"]).sum()
