"""A drop-in force call after the context's first mdg_set_state works on the centres it is given."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.MDG_FP64, abi.MDG_MIXED])
def test_centres_after_set_state(precision, gpulib):
    s, prm = configs.bulk_water()
    prm.precision = precision
    moved = s.copy()
    moved.c[0] += 0.01 * np.random.default_rng(3).standard_normal(moved.c[0].shape)
    moved.config_init()
    moved.rsx_after_predict()
    fresh = abi.Context(gpulib, s.copy(), prm)
    want = fresh.force_get(moved.copy())
    fresh.close()
    ctx = abi.Context(gpulib, s.copy(), prm)
    ctx.force_get(s.copy())
    ctx.set_state(ctx.sys)
    got = ctx.force_get(moved.copy())
    bar = 1e-5 if precision == abi.MDG_MIXED else 1e-12
    for k in ("fc", "torque"):
        assert np.linalg.norm(got[k] - want[k]) <= bar * np.linalg.norm(want[k]), k
    ctx.close()
