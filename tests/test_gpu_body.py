"""A later mdg_set_state with another thermostat or molecule steps with those, not with the ones of the run before."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.MDG_FP64, abi.MDG_MIXED])
@pytest.mark.parametrize("change", ["thermostat", "inertia"])
def test_second_state(precision, change, gpulib):
    s, prm = configs.bulk_water()
    prm.precision = precision
    other = s.copy()
    if change == "thermostat":
        other.temper = 250.0
    else:
        other.inxx, other.inyy = 1.1 * s.inxx, 1.2 * s.inyy
    pos = []
    for first in (s, None):
        ctx = abi.Context(gpulib, s.copy(), prm)
        if first is not None:
            ctx.set_state(first)
            ctx.run(2)
        got = other.copy()
        ctx.set_state(got)
        rep = ctx.run(8)
        ctx.get_state(got)
        pos.append((np.concatenate([got.c[0].ravel(), got.q[0].ravel()]), rep["kw"], got.s.copy()))
        ctx.close()
    a, b = pos
    # eight steps with forces added in another order: rounding of FP64, of FP32 in the mixed form
    bar = 1e-6 if precision == abi.MDG_MIXED else 1e-11
    assert np.abs(a[0] - b[0]).max() <= bar
    assert abs(a[1] - b[1]) <= bar * abs(b[1])
    assert np.abs(a[2] - b[2]).max() <= 100.0 * bar * np.abs(b[2]).max()
