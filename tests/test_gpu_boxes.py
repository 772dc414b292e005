"""Rectangular boxes: every form of the reciprocal sum with three different edges, the long one in each direction in
turn, against the oracle's direct sum; and edges long enough that the tables of a form do not fit, where another
form or smaller tables have to take the box as before.

Ions of random charges on a jittered lattice with no pair inside the cutoff: the forces are the reciprocal ones.
Bars: FP64 1e-12 of the forces' norm and of the energies' size, those of the cubic boxes; mixed 1e-5."""
import ctypes as C

import numpy as np
import pytest

from md_sim_gb300 import abi, configs
from md_sim_gb300 import system as S

pytestmark = pytest.mark.gpu


def ions(nx, ny, nz, kmax, precision, spacing=2.8):
    n = nx * ny * nz
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    box = spacing * np.array([nx, ny, nz])
    rng = np.random.default_rng(nx + 100 * ny + 10000 * nz)
    pos = rng.permutation(g * spacing + rng.uniform(-0.3, 0.3, (n, 3)) - 0.5 * box)
    kinds = [S.MolType(m, "atmol", n // 2, [m], [1], [0.03], [q], ns=1) for m, q in (("Na", 1.0), ("Cl", -1.0))]
    crys = S.MolType("none", "crystal", 1, ["X1", "X2"], [1, 1], [1e-3, 1e-3], [0.0, 0.0], ns=0, cx=box[0], cy=box[1], cz=box[2], lw=box[2])
    vdw = configs._vdw_table(["Na", "Cl", "X1", "X2"], {})
    s = S.System(S.FieldFile(kinds + [crys], vdw), S.TopFile([], [], [], []), *box, 1.0)
    s.x0[:n], s.y0[:n], s.z0[:n] = pos.T
    s.temper = -1.0
    return s, abi.RunParams(rcut=0.3, skin=0.1, kmax=kmax, alpha=0.35, variant=abi.MDG_BULK, pbc_z_list=1, precision=precision)


def compare(s, prm, gpulib, oracle):
    g, r = abi.Context(gpulib, s.copy(), prm), abi.Context(oracle, s.copy(), prm)
    b = r.force_get(s.copy())
    bar = 1e-5 if prm.precision == abi.MDG_MIXED else 1e-12
    for a in (g.force_get(s.copy()), g.force_get(s.copy())):
        assert np.linalg.norm(a["f"] - b["f"]) <= bar * np.linalg.norm(b["f"])
        for k in ("uewa", "ewqLL"):
            assert abs(a[k] - b[k]) <= bar * abs(b["uewa"]), k
    g.close()
    r.close()


EDGES = [(8, 12, 16), (16, 8, 12), (12, 16, 8)]


@pytest.mark.parametrize("edges", EDGES)
@pytest.mark.parametrize("precision,scale,kmax", [
    (abi.MDG_FP64, 1, 6),      # direct sums: 1.5e6 products of ions and k vectors
    (abi.MDG_FP64, 1, 12),     # FP64 grid: 1.1e7
    (abi.MDG_MIXED, 1, 8),     # tensor cores
    (abi.MDG_MIXED, 2, 15),    # FP32 grid: 1.8e8
])
def test_three_edges(precision, scale, kmax, edges, gpulib, oracle):
    s, prm = ions(*(scale * n for n in edges), kmax, precision)
    compare(s, prm, gpulib, oracle)


def test_long_x(gpulib, oracle):
    """|l| up to 432: 32 atoms' phase factors take more shared memory than there is."""
    s, prm = ions(72, 2, 2, 12, abi.MDG_FP64)
    compare(s, prm, gpulib, oracle)
    with pytest.raises(abi.MdgError, match="MDG_E_UNSUPPORTED"):
        abi.Context(gpulib, s, abi.RunParams(**{**prm.__dict__, "precision": abi.MDG_MIXED}))


def test_long_x_without_allocation(gpulib):
    torch = pytest.importorskip("torch")
    s, prm = ions(72, 2, 2, 12, abi.MDG_FP64)
    n = s.nmove
    ctx = abi.Context(gpulib, s.copy(), abi.RunParams(**{**prm.__dict__}))
    want = ctx.force_get(s.copy())
    ctx.close()
    f = gpulib.so.mdg_recip_forces_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p] * 4 + [C.c_int64] + [C.c_double] * 4 + [C.c_int64] + [C.c_void_p] * 5
    d = [torch.tensor(np.array(a[:n]), dtype=torch.float64, device="cuda:0") for a in (s.x0, s.y0, s.z0, s.qs)]
    out = [torch.zeros(n, dtype=torch.float64, device="cuda:0") for _ in range(3)] + [torch.zeros(1, dtype=torch.float64, device="cuda:0")]
    torch.cuda.synchronize()
    rc = f(*(t.data_ptr() for t in d), n, s.lx, s.ly, s.lz, prm.alpha, prm.kmax, *(t.data_ptr() for t in out), None)
    assert rc == 0, gpulib.last_error(None)
    torch.cuda.synchronize()
    got = np.stack([t.cpu().numpy() for t in out[:3]])
    assert np.linalg.norm(got - want["f"]) <= 1e-12 * np.linalg.norm(want["f"])
    assert abs(out[3].item() - want["uewa"]) <= 1e-12 * abs(want["uewa"])


@pytest.mark.parametrize("precision", [abi.MDG_FP64, abi.MDG_MIXED])
def test_long_y(precision, gpulib, oracle):
    """31,744 ions, |m| up to 85, about the longest that is accepted: the y twiddles of the FP64 grid do not fit (direct
    sums), those of the FP32 grid do."""
    s, prm = ions(16, 124, 16, 11, precision)
    compare(s, prm, gpulib, oracle)
