"""Positions that are not numbers end a force call with MDG_E_NAN, in either form, also when the neighbour lists
are those of the positions before."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.MDG_FP64, abi.MDG_MIXED])
@pytest.mark.parametrize("which", ["ion", "water"])
def test_nan_height(precision, which, gpulib):
    s, prm = configs.slab_electrolyte()
    ctx = abi.Context(gpulib, s.copy(), abi.RunParams(**{**prm.__dict__, "precision": precision}))
    ctx.force_get(s.copy())
    bad = s.copy()
    bad.z0[s.nriga + 1 if which == "ion" else 3] = np.nan
    with pytest.raises(abi.MdgError, match="MDG_E_NAN"):
        ctx.force_get(bad)
    ctx.force_get(s.copy())  # and the next call is none the worse
    ctx.close()
