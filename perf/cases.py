"""The work this library is timed on: force calls, resident MD steps, SHAKE steps, Widom insertion
and replica batches through the public entry points, from 256 to 32,768 waters.

A case is a dict of plain values; `listed` gives the fixed ones, `draw` others of the same ranges,
`prepare` what a program has in hand before the call (system, context, pinned host arrays), `run`
one pass through the entry points, `work` the bytes and operations a pass cannot do without, and
`exact` the same outputs from float64 torch, written from the reference's formulas.

Kinds of pass:
  force   mdg_force_get on pinned host arrays (the drop-in call of a host integrator): forces on
          flexible atoms, centre-of-mass forces, torques, energies
  md      `steps` resident MD steps (predictor, forces, corrector) at 300 K and the frame a program
          then reads back; the state goes on from pass to pass
  shake   mdg_force_get and mdg_shake from given positions (surface molecules with constraints)
  widom   one mdg_widom call on a state whose forces are there
  batch   `steps` steps of a replica batch and every replica's frame
Results of mixed-precision contexts are FP32 quantities in FP64 arrays (FP32 pair arithmetic) and
are returned as float32; plain FP64 contexts return float64.
"""
import ctypes as C
import math

import numpy as np
import torch

import md_sim_gb300
from md_sim_gb300 import abi, configs

SPACING = 3.103  # A per water of the bulk lattices (1 g/cm^3)
CELL = 4.21      # A, rocksalt wall cell


def listed():
    return [
        # the smallest box of the repository's configurations: latency and launches are the cost
        {"name": "force_bulk256_fp64", "kind": "force", "system": "fcc", "n": 4, "kmax": 7, "precision": "fp64"},
        {"name": "force_bulk256_mixed", "kind": "force", "system": "fcc", "n": 4, "kmax": 7, "precision": "mixed"},
        # the plain FP64 form: an interfacial slab, and the largest box
        {"name": "force_slab2048_fp64", "kind": "force", "system": "slab", "n": 2048, "cells": 10, "kmax": 10, "precision": "fp64"},
        {"name": "force_bulk32k_fp64", "kind": "force", "system": "sc", "n": 32, "kmax": 24, "precision": "fp64"},
        # the drop-in call at the largest box, and on a small slab with ions of odd counts
        {"name": "force_bulk32k_mixed", "kind": "force", "system": "sc", "n": 32, "kmax": 24, "precision": "mixed"},
        {"name": "force_ions517_mixed", "kind": "force", "system": "ions", "n": 517, "pairs": 19, "cells": 6, "kmax": 6, "precision": "mixed"},
        # production MD: an ordinary box of odd edge, the interfacial slab, the largest box
        {"name": "md_bulk2197_mixed", "kind": "md", "system": "sc", "n": 13, "kmax": 10, "precision": "mixed", "steps": 20},
        {"name": "md_slab2048_mixed", "kind": "md", "system": "slab", "n": 2048, "cells": 10, "kmax": 10, "precision": "mixed", "steps": 20},
        {"name": "md_bulk32k_mixed", "kind": "md", "system": "sc", "n": 32, "kmax": 24, "precision": "mixed", "steps": 20},
        # constrained waters on wide walls: force call and SHAKE, as a host's Verlet loop makes them
        {"name": "shake4913_mixed", "kind": "shake", "system": "shake", "n": 4913, "cells": 15, "kmax": 15, "precision": "mixed"},
        # chemical potential of water in the slab
        {"name": "widom_slab2048_fp64", "kind": "widom", "system": "slab", "n": 2048, "cells": 10, "kmax": 10, "precision": "fp64", "insertions": 2000},
        # many uneven interfacial replicas stepped together
        {"name": "batch16_mixed", "kind": "batch", "system": "slab", "replicas": 16, "mix": 5, "precision": "mixed", "steps": 20},
    ]


def draw(rng):
    kind = rng.choice(["force", "force", "force", "md", "md", "shake", "widom", "batch"])
    precision = rng.choice(["mixed", "mixed", "fp64"]) if kind in ("force", "md") else "fp64" if kind == "widom" else "mixed"
    if kind == "batch":
        return {"kind": kind, "system": "slab", "replicas": rng.randint(3, 16), "mix": rng.randint(1, 10 ** 6), "precision": precision, "steps": rng.randint(5, 20)}
    system = {"shake": "shake", "widom": "slab"}.get(kind) or rng.choice(["sc", "sc", "slab", "ions" if kind == "force" else "slab"])
    case = {"kind": kind, "system": system, "precision": precision}

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if system == "sc":
        # one evaluation in plain FP64 takes 0.1 s at n = 32: MD in that form stays smaller
        n = max(7, min(32, round(log_int(343, 32768 if precision == "mixed" or kind == "force" else 6000) ** (1 / 3))))
        case.update(n=n, kmax=round(n * SPACING * rng.uniform(0.235, 0.30)))
    else:
        n = log_int(300, {"shake": 4913, "ions": 2000}.get(system, 4000))
        cells = _cells(n, 6, rng.randint(7, 19), 60.0)
        case.update(n=n, cells=cells, kmax=round(10 * cells * CELL / 42.1 * rng.uniform(0.9, 1.1)))
    if system == "ions":
        case["pairs"] = rng.randint(3, 40)
    if kind == "md":
        case["steps"] = rng.randint(5, 20) if precision == "mixed" else rng.randint(1, 3)
    if kind == "widom":
        case["insertions"] = log_int(100, 2000)
    return case


def _cells(n, least, wanted, thickest):
    """Wall cells near `wanted` that keep a film of n waters between 20 A and `thickest`."""
    film = lambda cells: n / ((cells * CELL) ** 2 * 0.033427)  # noqa: E731
    while wanted > least and film(wanted) < 20.0:
        wanted -= 1
    while film(wanted) > thickest:
        wanted += 1
    return wanted


# ---- inputs ------------------------------------------------------------------------------------
def _system(case, seed):
    """(System, RunParams) of one case: the repository's synthetic systems from `seed`; lattices
    are jittered so that no two seeds share positions."""
    kind, system, n, kmax = case["kind"], case["system"], case["n"], case["kmax"]
    if system == "fcc":
        s, prm = configs.bulk_water(n, "fcc", seeds=(seed, seed + 1, seed + 2), kmax=kmax)
    elif system == "sc":
        s, prm = configs.bulk_water(n, "sc", box=n * SPACING, seeds=(seed, seed + 1, seed + 2), rcut=10.0 if n > 7 else 9.0,
                                    alpha=0.32, kmax=kmax)
    elif system == "slab":
        s, prm = configs.slab_water(n, case["cells"], lz=case.get("lz"), seed=seed, kmax=kmax, placement="lattice")
    elif system == "ions":
        s, prm = configs.slab_electrolyte(n, case["pairs"], case["cells"], seed=seed, kmax=kmax)
    else:
        s, prm = configs.shake_water(n, case["cells"], seed=seed, kmax=kmax)
    if system in ("fcc", "sc"):
        s.c[0] += np.random.default_rng(seed + 5).uniform(-0.15, 0.15, s.c[0].shape)
        s.config_init()
        s.rsx_after_predict()
    if kind in ("md", "batch"):
        _calm(s, seed)
    prm.precision = abi.MDG_MIXED if case["precision"] == "mixed" else abi.MDG_FP64
    return s, prm


def _calm(s, seed):
    """A start that production MD can go on from: no molecule within 3 A of a wall plane or turned
    into a neighbour, slow at first (the lattice's energy heats it), and the thermostat at 300 K."""
    if s.nwall:
        most = np.abs(s.c[0, 2]).max()
        s.c[0, 2] *= min(1.0, (s.lwh - 3.0) / most)
        n = slice(s.nriga, s.nliqa)
        s.z0[n] *= min(1.0, (s.lwh - 3.0) / most)
        fixed = np.stack([a[s.nriga:] for a in (s.x0, s.y0, s.z0)], 1)
        body = np.stack([s.xbody, s.ybody, s.zbody], 1)
        s.q[0] = configs._relax_orientations(np.random.default_rng(seed + 9), s.c[0].T, s.q[0], body, s.lx, s.lz, fixed, dmin=1.6)
    s.c[1] *= 0.3
    s.w[0] *= 0.3
    wx, wy, wz = s.w[0]
    q1, q2, q3, q4 = s.q[0]
    s.q[1] = 0.5 * np.stack([-q3 * wx - q4 * wy + q2 * wz, q4 * wx - q3 * wy - q1 * wz,
                             q1 * wx + q2 * wy + q4 * wz, -q2 * wx + q1 * wy - q3 * wz])
    s.config_init()
    s.rsx_after_predict()
    s.temper = 300.0


def _replicas(case, seed):
    """Uneven slabs: 500 to 4,000 waters on 6 to 14 wall cells, their sizes part of the case."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for k in range(case["replicas"]):
        n = int(rng.integers(500, 4001))
        cells = _cells(n, 6, int(rng.integers(7, 15)), 95.0)
        film = n / ((cells * CELL) ** 2 * 0.033427)
        one = {"kind": "batch", "system": "slab", "n": n, "cells": cells, "lz": max(2.0 * cells * CELL, film + 35.0),
               "kmax": round(10 * cells * CELL / 42.1), "precision": case["precision"]}
        out.append(_system(one, seed * 100 + k))
    return out


class _Pool:
    """Host arrays of one state in one range pinned by mdg_pin_host, as a host program pins its
    module arrays once."""

    def __init__(self, lib, words):
        self.lib, self.used = lib, 0
        self.buf = np.zeros(words)
        self.at = self.buf.ctypes.data
        if lib.pin_host(self.at, self.buf.nbytes) != 0:
            raise RuntimeError((lib.last_error(None) or b"").decode())

    def take(self, *shape):
        n = int(np.prod(shape))
        a = self.buf[self.used:self.used + n].reshape(shape)
        self.used += n + (-n) % 16
        return a

    def __del__(self):
        self.lib.unpin_host(self.at)


def _ptr(a):
    return a.ctypes.data_as(abi.DP)


class _State:
    """A system, its context and the host arrays of its calls."""

    def __init__(self, case, s, prm):
        self.case, self.sys, self.lib = case, s, md_sim_gb300.load()
        self.dtype = torch.float32 if case["precision"] == "mixed" else torch.float64
        self.ctx = abi.Context(self.lib, s, prm)
        nm, nr, nflex, nsurf = s.nmove, s.nrig, s.nmove - s.nriga, s.ntota - s.nliqa
        self.pool = p = _Pool(self.lib, 3 * s.ntota + 12 * nm + 40 * max(nr, 1) + 6 * max(nflex, 1) + 6 * nsurf + 4 * s.nijt + 4096)
        self.x = p.take(3, s.ntota)
        self.x[:] = s.x0, s.y0, s.z0
        self.c = p.take(3, max(nr, 1))
        if nr:
            self.c[:] = s.c[0]
        self.rs = p.take(3, nm)
        self.rs[:] = s.rsx, s.rsy, s.rsz
        self.rs_first = self.rs[:, :3].copy()
        self.ft, self.fc, self.tq = p.take(3, max(nflex, 1)), p.take(3, max(nr, 1)), p.take(3, max(nr, 1))
        self.elj, self.eqq = p.take(s.nijt), p.take(s.nijt)
        self.e = abi.Energies()
        self.e.elj, self.e.eqq = _ptr(self.elj), _ptr(self.eqq)
        self.args = [_ptr(a) for b in (self.x, self.c, self.rs, self.ft, self.fc, self.tq) for a in b] + [None] * 3 + [C.byref(self.e)]
        if case["kind"] == "shake":
            self.start = np.concatenate([self.x, np.stack([s.xold, s.yold, s.zold])], 1)
            self.old = p.take(3, nsurf)
            self.tk, self.sweeps = C.c_double(), C.c_int32()
            self.shake_args = [_ptr(a) for b in (self.x, self.old, self.ft) for a in b] + [None, C.byref(self.tk), C.byref(self.sweeps)]
        if case["kind"] in ("md", "batch"):
            self.ctx.set_state(s)
            self.v, self.quat, self.w = p.take(3, max(nr, 1)), p.take(4, max(nr, 1)), p.take(3, max(nr, 1))
            # a frame: site positions, centres and their velocities, quaternions, angular velocities
            self.frame = st = abi.State()
            st.x0, st.y0, st.z0 = (_ptr(a) for a in self.x)
            (st.cx[0], st.cy[0], st.cz[0]), (st.cx[1], st.cy[1], st.cz[1]) = map(_ptr, self.c), map(_ptr, self.v)
            for k in range(4):
                st.q[k][0] = _ptr(self.quat[k])
            st.wx[0], st.wy[0], st.wz[0] = map(_ptr, self.w)

    def out(self, a):
        """A copy of a result array in the precision of its context."""
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dtype, copy=True)

    def force(self):
        s, e = self.sys, self.e
        self.rs[:, :3] = self.rs_first  # the call leaves other values there
        self.ctx._check(self.lib.force_get(self.ctx.h, *self.args))
        out = {"energies": self.out(np.array([e.uconf, e.uewa, e.urf, e.ulr, e.uself, e.ewqLL, e.ewqWL, e.ewqWW])),
               "elj": self.out(self.elj), "eqq": self.out(self.eqq)}
        if s.nmove > s.nriga:
            out["ft"] = self.out(self.ft)
        if s.nrig:
            out["fc"], out["torque"] = self.out(self.fc), self.out(self.tq)
        return out

    def read_frame(self, rep):
        s = self.sys
        self.ctx._check(self.lib.get_state(self.ctx.h, C.byref(self.frame)))
        return {"x": self.out(self.x[:, :s.nmove]), "c": self.out(self.c), "v": self.out(self.v), "q": self.out(self.quat),
                "w": self.out(self.w), "report": self.out(np.array([rep["kp"], rep["kw"], rep["htot"], rep["uconf"]]))}


class _Batch:
    def __init__(self, case, seed):
        self.parts = [_State(case, s, prm) for s, prm in _replicas(case, seed)]
        self.batch = abi.Batch(self.parts[0].lib, [p.ctx for p in self.parts])


def prepare(case, seed):
    if case["kind"] == "batch":
        return _Batch(case, seed)
    st = _State(case, *_system(case, seed))
    st.seed = seed
    if case["kind"] == "widom":
        st.force()
    return st


# ---- one pass ----------------------------------------------------------------------------------
def run(state):
    if isinstance(state, _Batch):
        reps = state.batch.run(state.parts[0].case["steps"])
        frames = [p.read_frame(r) for p, r in zip(state.parts, reps)]
        return {k: torch.cat([f[k].reshape(-1) for f in frames]) for k in frames[0]}
    case = state.case
    if case["kind"] == "force":
        return state.force()
    if case["kind"] == "md":
        return state.read_frame(state.ctx.run(case["steps"]))
    if case["kind"] == "shake":
        s = state.sys
        state.x[:] = state.start[:, :s.ntota]
        state.old[:] = state.start[:, s.ntota + s.nliqa:]
        out = state.force()
        state.ctx._check(state.lib.shake(state.ctx.h, *state.shake_args))
        out["x"], out["tkps"] = state.out(state.x[:, s.nliqa:s.nmove]), state.tk.value
        return out
    w = state.ctx.widom(case["insertions"], 1.0, 6.0, 10, 0, 14135621772.0 + 7919.0 * (state.seed % 1000003),
                        flags=abi.MDG_WIDOM_SKIP_OVERLAP)
    return {"pave": w["pave"], "inave": w["inave"], "done": w["done"]}


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    """Each input read and each output written once; 45 operations per site pair inside the cutoff
    (at 1 g/cm^3, each pair once), 100 per atom and 30 per k vector for the reciprocal sum (a fast
    transform does without the product of the two), 500 per molecule for an integrator step."""
    if case["kind"] == "batch":
        atoms, walls, nk, steps = case["replicas"] * 3 * 2250, case["replicas"] * 3600, case["replicas"] * 4500, case["steps"]
    else:
        waters = {"fcc": 4 * case["n"] ** 3, "sc": case["n"] ** 3}.get(case["system"], case["n"])
        atoms = 3 * waters + 2 * case.get("pairs", 0)
        film = case["system"] not in ("fcc", "sc")
        walls = 16 * case["cells"] ** 2 if film else 0
        nk = 2 * math.pi / 3 * case["kmax"] ** 3 * (2 if film else 1)
        steps = case.get("steps", 1)
    pairs = atoms * (0.1003 * 4 / 3 * math.pi * 10.0 ** 3 / 2)
    flops = steps * (45.0 * pairs + 100.0 * atoms + 30.0 * nk + (500.0 * atoms / 3 if "steps" in case else 0.0))
    if case["kind"] == "widom":
        turns = 10.0 * case["insertions"]  # about half of the positions overlap, 20 orientations each
        return {"bytes": 32.0 * (atoms + walls) + 40.0 * nk, "flops": turns * (3 * 20.0 * nk + 3 * 45.0 * 0.1003 * 4189)}
    if case["kind"] in ("md", "batch"):
        return {"bytes": 8.0 * (6 * atoms + 50 * atoms / 3) * 2, "flops": flops}
    n_in, n_out = (6 + 6, 3 + 6) if case["kind"] == "shake" else (7, 2)
    return {"bytes": 8.0 * (n_in + n_out) * atoms, "flops": flops}


# ---- the same in float64 torch --------------------------------------------------------------------
def _f32(x):
    """A single-precision literal of the reference, as it enters its double-precision arithmetic."""
    return float(np.float32(x))


PI = _f32(3.1415926535898)
R_GAS = _f32(8.31441)
E_CH, N_AV, EPS0, K_EL, ANG = _f32(1.6021892e-19), _f32(6.022045e23), _f32(8.85418782e-12), _f32(8.987551784952e9), _f32(1e-10)
ERF_A = [_f32(a) for a in (1.061405429, -1.453152027, 1.421413741, -0.284496736, 0.254829592)]
ERF_P = _f32(0.3275911)


class _Exact:
    """Forces and energies of one system (force_real, force_fouri, force_sum), in float64."""

    def __init__(self, s, prm):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.s, self.prm = s, prm
        t = lambda a, d=torch.float64: torch.as_tensor(np.array(a), dtype=d, device=self.dev)  # noqa: E731
        self.t = t
        self.box = [s.lx, s.ly, s.lz]
        self.slab = prm.variant == abi.MDG_SLAB
        self.alpha = prm.alpha
        self.q, self.typ = t(s.qs), t(s.itype, torch.long) - 1
        self.ijt = t(s.ijtype, torch.long).reshape(s.nit, s.nit) - 1
        nsi = t(s.nsi, torch.long)[self.typ[:s.nmove]]
        self.heads = torch.nonzero(nsi).flatten()
        self.nsi = nsi
        self.vdw = [t(s.vdwnum, torch.long)] + [t(a) for a in (s.eps, s.sig, s.aa, s.rhoi, s.cc)]
        self.facq = K_EL * E_CH * E_CH * N_AV / (1000.0 * ANG)
        self.spii = 2.0 / math.sqrt(PI)
        self.wall = t(np.stack([s.x0[s.nmove:], s.y0[s.nmove:], s.z0[s.nmove:]]))
        # molecule of each constrained atom: pairs held by a constraint do not interact
        mol = np.arange(s.ntota) + s.ncons
        for k in range(3 if s.ncons else 0):
            for tab in (s.constra, s.constrb):
                ok = tab[k] > 0
                mol[tab[k][ok] - 1] = np.arange(s.ncons)[ok]
        self.mol = t(mol, torch.long)
        self._k_set()
        self._tails()
        self._self_energy()

    def _image(self, d):
        for k in range(3 if not self.slab else 2):
            u = d[k] / self.box[k]
            d[k] -= self.box[k] * torch.sign(u) * torch.floor(u.abs() + 0.5)
        return d

    def _erfc(self, r):
        ar = self.alpha * r
        u = 1.0 / (1.0 + ERF_P * ar)
        g = torch.exp(-ar * ar)
        p = ERF_A[0]
        for a in ERF_A[1:]:
            p = p * u + a
        e = p * u * g
        return e, self.spii * ar * g + e

    def _vdw(self, k, r2):
        kind, eps, sig, aa, rhoi, cc = (v[k] for v in self.vdw)
        r = torch.sqrt(r2)
        i6 = 1.0 / r2 ** 3
        lj, bu = sig * i6, cc * i6
        ex = aa * torch.exp(-r * rhoi)
        u = torch.where(kind == 1, eps * lj * (lj - 1.0), torch.where(kind == 2, ex - bu, 0.0))
        f = torch.where(kind == 1, 6.0 / r2 * eps * lj * (2.0 * lj - 1.0), torch.where(kind == 2, ex * rhoi / r - 6.0 / r2 * bu, 0.0))
        return u, f

    def _near(self, a, b, own):
        """(i, j) of columns of a, b within the cutoff (own: i < j of one set)."""
        out, rows = [], max(1, (1 << 24) // max(b.shape[1], 1))
        for i0 in range(0, a.shape[1], rows):
            d = self._image([a[k, i0:i0 + rows, None] - b[k] for k in range(3)])
            near = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] <= self.prm.rcut ** 2
            p = torch.nonzero(near)
            p[:, 0] += i0
            out.append(p[p[:, 0] < p[:, 1]] if own else p)
        return torch.cat(out).T

    def _real(self, x, rs, f, elj, eqq):
        hd = self.heads
        if hd.numel() == 0:
            return
        h = x[:, hd]
        i, j = self._near(h, h, True)
        i, j = hd[i], hd[j]
        free = self.mol[i] != self.mol[j]
        i, j = i[free], j[free]
        d0 = torch.stack(self._image([x[k, i] - x[k, j] for k in range(3)]))
        r2 = (d0 * d0).sum(0)
        k = self.ijt[self.typ[i], self.typ[j]]
        u, fv = self._vdw(k, r2)
        elj.index_add_(0, k, u)
        ni, nj = self.nsi[i], self.nsi[j]
        for a in range(3):
            for b in range(3):
                on = (ni > a) & (nj > b)
                ia, jb = i[on] + a, j[on] + b
                if a == b == 0:
                    d, add = d0, fv
                else:
                    d, add = d0[:, on] + rs[:, ia] - rs[:, jb], 0.0
                rr = (d * d).sum(0)
                r = torch.sqrt(rr)
                c = self.facq * self.q[ia] * self.q[jb] / r
                e, g = self._erfc(r)
                eqq.index_add_(0, k[on], e * c)
                fp = d * (add + g * c / rr)
                f.index_add_(1, ia, fp)
                f.index_add_(1, jb, -fp)
        if not self.s.nwall:
            return
        i, w = self._near(h, self.wall, False)
        i = hd[i]
        d0 = torch.stack(self._image([x[k, i] - self.wall[k, w] for k in range(3)]))
        jw = w + self.s.nmove
        k = self.ijt[self.typ[i], self.typ[jw]]
        u, fv = self._vdw(k, (d0 * d0).sum(0))
        elj.index_add_(0, k, u)
        for a in range(3):
            on = self.nsi[i] > a
            ia = i[on] + a
            d = d0[:, on] + rs[:, ia]
            rr = (d * d).sum(0)
            r = torch.sqrt(rr)
            c = self.facq * self.q[jw[on]] * self.q[ia] / r
            e, g = self._erfc(r)
            eqq.index_add_(0, k[on], e * c)
            f.index_add_(1, ia, d * ((fv[on] if a == 0 else 0.0) + g * c / rr))

    def _tails(self):
        """force_real_init: the layers beyond the cutoff as continua, per site type."""
        s, rc = self.s, self.prm.rcut
        tab = np.zeros((9, s.nit))
        tab[6] = 1.0
        if self.slab:
            nstw = int(s.nst[s.ntype - 1])
            dens = np.bincount(s.itype[:s.nmove] - 1, minlength=s.nit).astype(float)
            dens[:s.nit - nstw] *= s.nmove / (s.lx * s.ly * s.lw) / s.nmove
            rho = s.nss_wall[:nstw].sum() / (2.0 * s.cx * s.cy * s.cz)
            dens[-2:] = [_f32(np.float32(n) / np.float32(s.nss_wall.sum())) * rho for n in s.nss_wall[:2]]
            ij = np.asarray(s.ijtype).reshape(s.nit, s.nit) - 1
            for it in range(s.nit - nstw):
                for jt in range(s.nit):
                    k, wall = ij[jt, it], jt >= s.nit - nstw
                    sg, e, g = (1.0 if wall else -1.0) * dens[jt], s.eps[k], s.sig[k]
                    fl = ul = 0.0
                    if s.vdwnum[k] == 1:
                        fl = e * g * (g / (10 * rc ** 10) - 1 / (4 * rc ** 4))
                        ul = e * g * (g / (90 * rc ** 9) - 1 / (12 * rc ** 3))
                        tab[2, it] += sg * e * g * g / 10
                        tab[3, it] += sg * e * g / 4
                    elif s.vdwnum[k] == 2:
                        ro = 1.0 / s.rhoi[k]
                        ex = s.aa[k] * math.exp(-rc / ro)
                        fl = ro * (ro + rc) * ex - s.cc[k] / (4 * rc ** 4)
                        ul = ro * ro * (2 * ro + rc) * ex - s.cc[k] / (12 * rc ** 3)
                        tab[4, it] += sg * s.aa[k] * ro
                        tab[5, it] += sg * s.cc[k] / 4
                        tab[6, it] = ro
                    tab[1 if wall else 0, it] += fl * dens[jt]
                    tab[8 if wall else 7, it] += ul * dens[jt]
            tab[[0, 1, 2, 3, 4, 5, 7, 8]] *= 2 * PI
        self.tab = self.t(tab)

    def _tail(self, x, f):
        if not self.slab:
            return 0.0
        n = self.s.nmove
        big = torch.nonzero(self.q[:n].abs() >= _f32(0.7)).flatten()
        z, u = x[2, big], 0.0
        fl, fw, lja, ljc, bua, buc, bur, ul, uw = (self.tab[k][self.typ[big]] for k in range(9))
        for sg in (-1.0, 1.0):
            d = 0.5 * self.s.lw - sg * z
            ex = bua * torch.exp(-d / bur)
            far = fl + lja / d ** 10 - ljc / d ** 4 + (bur + d) * ex - buc / d ** 4
            ufar = ul + lja / (9 * d ** 9) - ljc / (3 * d ** 3) + bur * (2 * bur + d) * ex - buc / (3 * d ** 3)
            near = d < self.prm.rcut
            f[2].index_add_(0, big, -sg * torch.where(near, fw, far))
            u += float(torch.where(near, uw, ufar).sum())
        return u

    def _k_set(self):
        s, kmax = self.s, self.prm.kmax
        lmin = min(self.box)
        K = [int(math.floor(kmax * b / lmin + 0.5)) for b in self.box]
        l, m, n = (np.arange(lo, k + 1) for lo, k in ((0, K[0]), (-K[1], K[1]), (-K[2], K[2])))
        L, M, N = np.meshgrid(l, m, n, indexing="ij")
        size = (L * L + M * M).astype(np.float32) + (N * N * kmax * kmax).astype(np.float32) / np.float32(K[2] ** 2)
        keep = (size < np.float32(kmax * kmax) + np.float32(2.01)) & ((L > 0) | (M > 0) | ((M == 0) & (N > 0)))
        g = [2 * PI / b for b in self.box]
        ksq = (g[0] * L) ** 2 + (g[1] * M) ** 2 + (g[2] * N) ** 2
        fac = 2.0 * E_CH * E_CH * N_AV / (EPS0 * ANG * 1000.0 * s.lx * s.ly * s.lz)
        ak = np.where(keep, fac * np.exp(-ksq / (4 * self.alpha ** 2)) / np.where(keep, ksq, 1.0), 0.0)
        self.ak, self.K, self.g, self.lmn = self.t(ak), K, g, [self.t(a) for a in (l, m, n)]
        self.qw = self._sfac(self.wall, self.q[s.nmove:]) if s.nwall else torch.zeros_like(self.ak, dtype=torch.complex128)
        self.ww = 0.5 * float((self.ak * (self.qw.abs() ** 2)).sum())

    def _phases(self, x):
        return [torch.polar(torch.ones((), dtype=torch.float64, device=self.dev), self.g[k] * x[k][:, None] * self.lmn[k]) for k in range(3)]

    def _sfac(self, x, q):
        S = torch.zeros(self.ak.shape, dtype=torch.complex128, device=self.dev)
        for i0 in range(0, x.shape[1], 16384):
            el, em, en = self._phases(x[:, i0:i0 + 16384])
            for k in range(el.shape[1]):
                S[k] += (q[i0:i0 + 16384, None] * el[:, k:k + 1] * em).T @ en
        return S

    def _recip(self, x, f):
        n, q = self.s.nmove, self.q[:self.s.nmove]
        S = self._sfac(x[:, :n], q)
        tot = S + self.qw
        coef = self.ak * tot.conj()
        for i0 in range(0, n, 16384):
            at = slice(i0, min(n, i0 + 16384))
            el, em, en = self._phases(x[:, at])
            for k in range(el.shape[1]):
                t = en @ coef[k].T
                tz = en @ (coef[k] * self.lmn[2]).T
                e = q[at, None] * el[:, k:k + 1] * em
                im = (e * t).imag
                f[0, at] += self.g[0] * self.lmn[0][k] * im.sum(1)
                f[1, at] += self.g[1] * (im * self.lmn[1]).sum(1)
                f[2, at] += self.g[2] * (e * tz).imag.sum(1)
        u, ll = (0.5 * float((self.ak * a.abs() ** 2).sum()) for a in (tot, S))
        if not self.slab:
            return u, ll, 0.0
        dip = float((q * x[2, :n]).sum())
        crf = -2.0 * PI / (self.s.lx * self.s.ly * self.s.lz)
        f[2] += 2.0 * crf * self.facq * dip * q
        return u, ll, -crf * self.facq * dip * dip

    def _self_energy(self):
        s = self.s
        u = -0.5 * self.spii * self.facq * self.alpha * float((s.qs ** 2).sum())
        erf = lambda r: 1.0 - float(self._erfc(torch.tensor(r, dtype=torch.float64))[0])  # noqa: E731
        first, seen = 0, 0
        for it in range(s.ntype):
            if s.moltypen[it] == 0:
                at = range(first, first + int(s.ns[it]))
                for a in at:
                    for b in at:
                        if a < b:
                            r = math.dist((s.x0[a], s.y0[a], s.z0[a]), (s.x0[b], s.y0[b], s.z0[b]))
                            u -= float(s.nt[it]) * self.facq * s.qs[a] * s.qs[b] * erf(r) / r
            elif s.moltypen[it] == 2:
                # the reference reads its (3, ncons) tables transposed here
                fa, fb = s.constra.flatten(order="F"), s.constrb.flatten(order="F")
                for iq in range(int(s.nt[it])):
                    for k in range(int(s.nconst[it])):
                        at = seen + iq + 3 * k
                        if at < fa.size and fa[at] > 0 and fb[at] > 0:
                            u -= self.facq * s.qs[fa[at] - 1] * s.qs[fb[at] - 1] * self._erf_of(it, k, erf)
                seen += int(s.nt[it])
            first = int(s.nt[it])
        self.uself = u

    def _erf_of(self, it, k, erf):
        if not hasattr(self, "_bonds"):
            self._bonds = {}
        if (it, k) not in self._bonds:
            r = float(self.s.length[it, k])
            self._bonds[it, k] = erf(r) / r
        return self._bonds[it, k]

    def force(self, x, c, rs):
        s = self.s
        f = torch.zeros(3, s.nmove, dtype=torch.float64, device=self.dev)
        elj, eqq = torch.zeros(2, s.nijt, dtype=torch.float64, device=self.dev)
        self._real(x, rs, f, elj, eqq)
        ulr = self._tail(x, f)
        uewa, ll, urf = self._recip(x, f)
        uconf = float(elj.sum() + eqq.sum()) + uewa + urf
        out = {"energies": self.t([uconf, uewa, urf, ulr, self.uself, ll, uewa - self.ww - ll, self.ww]), "elj": elj, "eqq": eqq}
        if s.nmove > s.nriga:
            out["ft"] = f[:, s.nriga:]
        if s.nrig:
            site, arm = f[:, :s.nriga].reshape(3, -1, 3), x[:, :s.nriga].reshape(3, -1, 3) - c[:, :, None]
            out["fc"], out["torque"] = site.sum(2), torch.linalg.cross(arm, site, dim=0).sum(2)
        return out


G1 = [_f32(0.348611111), 1.0, _f32(0.916666667), _f32(0.333333333), _f32(0.041666667)]  # first-order equations
G2 = [_f32(0.1583), _f32(0.757), 1.0, 0.5, _f32(0.083333333)]                           # second-order
TAYLOR = np.array([[1.0, 1, 1, 1, 1], [0, 1, 2, 3, 4], [0, 0, 1, 3, 6], [0, 0, 0, 1, 4], [0, 0, 0, 0, 1]])


def _exact_md(s, prm, steps):
    """The Gear steps of rigid molecules and ions with the reference's two thermostats, in float64."""
    E = _Exact(s, prm)
    t = E.t
    nr, na, nl = s.nrig, s.nriga, s.nliqa
    x = t(np.stack([s.x0, s.y0, s.z0]))
    rs = t(np.stack([s.rsx, s.rsy, s.rsz]))
    ion = torch.cat([x[None, :, na:nl], t(s.xd[:, :, na:nl])])
    c, q, w, th, tr = (t(a) for a in (s.c, s.q, s.w, s.s, s.rs))
    body = t(np.stack([s.xbody, s.ybody, s.zbody]))
    inert = t([s.inxx, s.inyy, s.inzz])[:, None]
    up, g1, g2 = t(TAYLOR), t(G1)[:, None, None], t(G2)[:, None, None]
    mi, mii = t(s.mi)[na:nl], t(s.mii)[na:nl]
    nfree, nvt, uconf = nl - na, s.temper != -1.0, 0.0
    tstar = R_GAS * s.temper / 1000.0
    qmass, rmass = 3 * (nfree + nr) * tstar * 200.0, 3 * nr * tstar * 100.0
    ahead = lambda a: torch.tensordot(up, a, dims=1)  # noqa: E731
    for _ in range(steps):
        ion, c, q, w = ahead(ion), ahead(c), ahead(q), ahead(w)
        kp = float((mi * (ion[1] ** 2).sum(0)).sum() + s.mw * (c[1] ** 2).sum())
        kw = float((inert * w[0] ** 2).sum())
        q[0] = q[0] / torch.sqrt((q[0] ** 2).sum(0))
        q1, q2, q3, q4 = q[0]
        rot = torch.stack([torch.stack([-q1 * q1 + q2 * q2 - q3 * q3 + q4 * q4, 2 * (q3 * q4 - q1 * q2), 2 * (q2 * q3 + q1 * q4)]),
                           torch.stack([-2 * (q1 * q2 + q3 * q4), q1 * q1 - q2 * q2 - q3 * q3 + q4 * q4, 2 * (q2 * q4 - q1 * q3)]),
                           torch.stack([2 * (q2 * q3 - q1 * q4), -2 * (q1 * q3 + q4 * q2), -q1 * q1 - q2 * q2 + q3 * q3 + q4 * q4])])
        site = c[0][:, :, None] + torch.einsum("bdm,bj->dmj", rot, body)
        x[:, :na] = site.reshape(3, -1)
        x[:, na:nl] = ion[0]
        off = rs[:, :na].reshape(3, nr, 3)
        off[:, :, 1:] = site[:, :, 1:] - site[:, :, :1]
        if nvt:
            th, tr = up @ th, up @ tr
        else:
            th[:2] = tr[:2] = 0.0
        htot = 0.5 * (kp + kw + qmass * float(th[0]) ** 2 + rmass * float(tr[0]) ** 2) + uconf
        out = E.force(x, c[0], rs)
        rs[:, :3] = site[:, -1] - c[0][:, -1:]  # force_sum leaves the last molecule's arms there
        uconf = float(out["energies"][0])
        if nfree:
            ion = ion + g2 * (0.5 * out["ft"][:, :nfree] * mii - ion[1] * th[0] - ion[2])
        c = c + g2 * (0.5 / s.mw * out["fc"] - c[1] * th[0] - c[2])
        wx, wy, wz = w[0]
        dq = 0.5 * torch.stack([-q3 * wx - q4 * wy + q2 * wz, q4 * wx - q3 * wy - q1 * wz,
                                q1 * wx + q2 * wy + q4 * wz, -q2 * wx + q1 * wy - q3 * wz])
        q = q + g1 * (dq - q[1])
        i1, i2, i3 = inert
        gyro = torch.stack([wy * wz * (i2 - i3), wz * wx * (i3 - i1), wx * wy * (i1 - i2)])
        w = w + g1 * ((torch.einsum("bdm,dm->bm", rot, out["torque"]) + gyro) / inert - w[1] - tr[0] * w[0])
        if nvt:
            for v, rate in ((th, (kp - (3 * (nfree + nr) - 2) * tstar) / qmass), (tr, (kw - (3 * nr + 1) * tstar) / rmass)):
                d = rate - float(v[1])
                v += t(G1) * d
                v[1] = rate
    x[:, na:nl] = ion[0]
    return {"x": x[:, :s.nmove], "c": c[0], "v": c[1], "q": q[0].contiguous(), "w": w[0], "report": t([kp, kw, htot, uconf])}


def _exact_shake(s, prm, E, out):
    """Verlet step of the surface atoms, then the constraint sweeps in the reference's order."""
    t, nl, nm = E.t, s.nliqa, s.nmove
    x, old = t(np.stack([s.x0, s.y0, s.z0]))[:, nl:nm], t(np.stack([s.xold, s.yold, s.zold]))[:, nl:nm]
    d = x - old
    for k in range(2):
        d[k] -= E.box[k] * torch.round(d[k] / E.box[k])
    kin = float((t(s.mi)[nl:nm] * (d * d).sum(0)).sum())
    mii = t(s.mii)[nl:nm]
    new = x + d + out["ft"][:, nl - s.nriga:] * mii
    ia, ib = (t(a, torch.long) - 1 - nl for a in (s.constra, s.constrb))
    length = t(s.length)[t(s.ictype, torch.long) - 1].T
    for _ in range(prm.shake_maxit):
        worst = 0.0
        for k in range(3):
            a, b = ia[k], ib[k]
            p, r = new[:, a] - new[:, b], x[:, a] - x[:, b]
            for v in (p, r):
                for ax in range(3):
                    v[ax] -= E.box[ax] * torch.round(v[ax] / E.box[ax])
            diff = length[k] ** 2 - (p * p).sum(0)
            worst = max(worst, float((diff.abs() / length[k] ** 2).max()))
            g = diff / (2.0 * (mii[a] + mii[b]) * (r * p).sum(0))
            new[:, a] += r * g * mii[a]
            new[:, b] -= r * g * mii[b]
        if worst < 1e-14:
            break
    free = 3 * (nm - nl) - int(sum(s.nt[k] * s.nconst[k] for k in range(s.ntype) if s.moltypen[k] == 2))
    return {**out, "x": new, "tkps": kin * 1000.0 / (R_GAS * free)}


def exact(case, seed):
    if case["kind"] == "widom":
        return None  # a sum over some 20,000 trial energies, each over all k vectors and sites
    if case["kind"] == "batch":
        if case["replicas"] * case["steps"] > 120:
            return None  # over 20 s
        frames = [_exact_md(s, prm, case["steps"]) for s, prm in _replicas(case, seed)]
        return {k: torch.cat([f[k].reshape(-1) for f in frames]) for k in frames[0]}
    s, prm = _system(case, seed)
    if case["kind"] == "md":
        return _exact_md(s, prm, case["steps"])
    E = _Exact(s, prm)
    out = E.force(E.t(np.stack([s.x0, s.y0, s.z0])), E.t(s.c[0]), E.t(np.stack([s.rsx, s.rsy, s.rsz])))
    return _exact_shake(s, prm, E, out) if case["kind"] == "shake" else out
