"""Allocations that fail, one after the other (MDG_DEBUG_FAIL_ALLOC: the n-th of a context, on the host): a call that
does without one of its arrays says so, and nothing runs on an array that is not there."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "fp64 direct": (abi.MDG_FP64, lambda: configs.slab_water(96, 6, kmax=6, placement="lattice")),
    "fp64 gridded": (abi.MDG_FP64, lambda: configs.slab_water(700, 7, kmax=12, placement="lattice")),
    "mixed": (abi.MDG_MIXED, lambda: configs.slab_water(96, 6, kmax=6, placement="lattice")),
    "mixed gridded": (abi.MDG_MIXED, lambda: configs.slab_water(64, 6, kmax=6, lz=6 * 4.21 * 5.6, placement="lattice")),
}
MOST = 130  # more than a context's creation asks for


def _system(name):
    precision, make = SYSTEMS[name]
    s, prm = make()
    prm.precision = precision
    return s, prm


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_creation(name, gpulib, monkeypatch):
    """Every allocation of mdg_create in turn: no context, or (where the direct FP64 sums take the place of the
    gridded one) a context that works."""
    s, prm = _system(name)
    ref = abi.Context(gpulib, s.copy(), prm)
    a = ref.force_get(s.copy())["f"]
    ref.close()
    refused = []
    for n in range(1, MOST):
        monkeypatch.setenv("MDG_DEBUG_FAIL_ALLOC", str(n))
        try:
            ctx = abi.Context(gpulib, s.copy(), prm)
        except abi.MdgError as e:
            assert abi.ERRORS[e.code] == "MDG_E_CUDA", e
            refused.append(n)
            continue
        # the bars of the two forms against the oracle, of either sum
        bar = 1e-5 if prm.precision == abi.MDG_MIXED else 2e-12
        b = ctx.force_get(s.copy())["f"]
        assert np.linalg.norm(b - a) <= bar * np.linalg.norm(a), n
        ctx.close()
    assert len(refused) > 60 and refused[-1] < MOST - 5
    assert name == "fp64 gridded" or refused == list(range(1, len(refused) + 1))


@pytest.mark.parametrize("name", ["fp64 direct", "mixed"])
def test_widom(name, gpulib, monkeypatch):
    """Every allocation of the first insertion call in turn: it reports the failure, and the next call inserts as
    if nothing had been."""
    s, prm = _system(name)

    def insert(ctx):
        return ctx.widom(20, 1.0, 4.0, 8, 0, 14135621772.0, flags=abi.MDG_WIDOM_SKIP_OVERLAP)

    ctx = abi.Context(gpulib, s.copy(), prm)
    ctx.force_get(s.copy())
    want = insert(ctx)
    ctx.close()
    failed = 0
    for n in range(1, MOST):
        monkeypatch.setenv("MDG_DEBUG_FAIL_ALLOC", str(n))
        try:
            ctx = abi.Context(gpulib, s.copy(), prm)
        except abi.MdgError:
            continue
        ctx.force_get(s.copy())
        try:
            got = insert(ctx)
        except abi.MdgError as e:
            assert "out of memory" in str(e)
            failed += 1
            got = insert(ctx)
        assert got["seed"] == want["seed"] and got["done"] == want["done"]
        np.testing.assert_array_equal(got["inave"], want["inave"])
        # sums in another order, of energies with atomically added terms
        assert np.abs(got["pave"] - want["pave"]).max() <= (1e-4 if name == "mixed" else 1e-9) * want["pave"].max()
        ctx.close()
    assert failed == 7  # six arrays and the pinned staging


@pytest.mark.parametrize("name", ["fp64 direct", "mixed"])
def test_resident_state(name, gpulib, monkeypatch):
    """Every allocation of the first mdg_set_state in turn: it reports the failure, and the next one starts a run like
    any other."""
    s, prm = _system(name)
    ctx = abi.Context(gpulib, s.copy(), prm)
    ctx.set_state(ctx.sys)
    ctx.run(2)
    ctx.get_state()
    want = ctx.sys.x0.copy()
    ctx.close()
    failed = 0
    for n in range(1, MOST):
        monkeypatch.setenv("MDG_DEBUG_FAIL_ALLOC", str(n))
        try:
            ctx = abi.Context(gpulib, s.copy(), prm)
        except abi.MdgError:
            continue
        try:
            ctx.set_state(ctx.sys)
        except abi.MdgError as e:
            assert "out of device memory" in str(e)
            failed += 1
            ctx.force_get(ctx.sys.copy())  # the drop-in call goes on as before
            ctx.set_state(ctx.sys)
        ctx.run(2)
        ctx.get_state()
        # atomically added forces: rounding of FP64, of FP32 in the mixed form
        assert np.abs(ctx.sys.x0 - want).max() <= (1e-7 if name == "mixed" else 1e-11) * s.lx
        ctx.close()
    assert failed == 10  # the pinned thermostat values, eight arrays and the snapshot


@pytest.mark.parametrize("precision", [abi.MDG_FP64, abi.MDG_MIXED])
def test_list_growth(precision, gpulib, monkeypatch):
    """A force call whose lists outgrow their room and find no memory: it says so, and the next call has them."""
    s, prm = configs.ion_lattice(6, rcut=3.5, shuffle=True)
    prm.precision, prm.list_capacity = precision, 1
    near = s.copy()
    for a in (near.x0, near.y0, near.z0):
        a[:s.nmove] *= 0.4
    ctx = abi.Context(gpulib, s.copy(), prm)
    want = ctx.force_get(near.copy())["f"]
    ctx.close()
    failed = 0
    for n in range(1, MOST):
        monkeypatch.setenv("MDG_DEBUG_FAIL_ALLOC", str(n))
        try:
            ctx = abi.Context(gpulib, s.copy(), prm)
        except abi.MdgError:
            continue
        try:
            got = ctx.force_get(near.copy())
        except abi.MdgError as e:
            assert "out of device memory" in str(e)
            failed += 1
            got = ctx.force_get(near.copy())
        assert np.linalg.norm(got["f"] - want) <= (1e-5 if precision else 1e-12) * np.linalg.norm(want)
        ctx.close()
    assert failed == 2
