"""A replica that changes between two runs of its batch (another thermostat; lists that a call of its own made grow)
goes on as the same system alone does, in both graph forms."""
import numpy as np
import pytest

from md_sim_gb300 import abi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [abi.MDG_BATCH_PHASES, abi.MDG_BATCH_GRAPHS])
@pytest.mark.parametrize("precision", [abi.MDG_FP64, abi.MDG_MIXED])
@pytest.mark.parametrize("change", ["thermostat", "lists"])
def test_replica_changes(change, precision, mode, gpulib):
    def contexts():
        out = []
        for k in range(2):
            s, p = configs.slab_water(nwat=256 + 64 * k, cells=6, seed=40 + k, kmax=6, placement="lattice")
            p.precision, p.list_capacity = precision, 1
            out.append(abi.Context(gpulib, s, p))
            out[-1].set_state(s)
        return out

    def alter(c):
        c.get_state()
        if change == "thermostat":
            c.sys.temper = 200.0
        else:
            near = c.sys.copy()
            near.c[0] *= 0.6
            near.config_init()
            near.rsx_after_predict()
            c.force_get(near)
        c.set_state(c.sys)

    together, alone = contexts(), contexts()
    batch = abi.Batch(gpulib, together)
    batch.set_mode(mode)
    batch.run(3)
    alter(together[0])
    reps = batch.run(6)
    alone[0].run(3)
    alter(alone[0])
    alone[1].run(3)
    # forces added in another order, from the same start: the bars of the other batch tests
    bar = 1e-7 if precision == abi.MDG_MIXED else 1e-9
    for c, d, r in zip(together, alone, reps):
        one = d.run(6)
        c.get_state()
        d.get_state()
        assert np.abs(c.sys.x0 - d.sys.x0).max() < bar * c.sys.lx
        assert np.abs(c.sys.s - d.sys.s).max() <= 1e4 * bar * np.abs(d.sys.s).max()
        assert abs(r["uconf"] - one["uconf"]) <= 1e-5 * abs(one["uconf"])
    batch.close()
