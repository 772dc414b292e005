"""Mixed form with k vectors far beyond what the sum needs."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmax", [20, 24, 31])
def test_coefficients_beyond_fp32(kmax, gpulib, oracle):
    """k vectors so long that their coefficients are subnormal or zero in FP32: they count for nothing."""
    s, prm = configs.bulk_water(kmax=kmax)
    out = []
    for lib, p in ((gpulib, abi.MDG_MIXED), (oracle, abi.MDG_FP64)):
        ctx = abi.Context(lib, s.copy(), abi.RunParams(**{**prm.__dict__, "precision": p}))
        out.append(ctx.force_get(s.copy()))
        ctx.close()
    a, b = out
    assert np.linalg.norm(a["f"] - b["f"]) <= 1e-5 * np.linalg.norm(b["f"])
