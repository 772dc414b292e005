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


def test_few_atoms_many_k(gpulib):
    """1,536 atoms and 62,519 k vectors, above the line of the gridded sum but 1,500 grid points per atom: the
    tensor-core sum, in as many kernels as with few k vectors, and its forces."""
    kernels = []
    for kmax in (6, 31):
        s, prm = configs.bulk_water(8, "sc", box=24.824, kmax=kmax)
        out = []
        for p in (abi.MDG_FP64, abi.MDG_MIXED):
            ctx = abi.Context(gpulib, s.copy(), abi.RunParams(**{**prm.__dict__, "precision": p}))
            out.append(ctx.force_get(s.copy())["f"])
            if p == abi.MDG_MIXED:
                ctx.set_state(ctx.sys)
                ctx.run(1)
                kernels.append(ctx.kernels_per_step())
            ctx.close()
        assert np.linalg.norm(out[1] - out[0]) <= 1e-5 * np.linalg.norm(out[0])
    assert kernels[0] == kernels[1]
