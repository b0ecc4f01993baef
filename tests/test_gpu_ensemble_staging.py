"""Ensembles whose members stage different amounts of shared memory in one
group: with 16^2 tiles an FP64 tile of 16 fields stages more than one of 20,
so the group's launches are sized by the largest staging, not by the member
with the most fields."""
import numpy as np
import pytest

from w3914777_gb300 import amps, ensemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fields", [(20, 16), (17, 9, 16, 27), (24, 3, 16)])
@pytest.mark.parametrize("ref_order", [0, 1])
def test_members_of_one_group_equal_their_single_runs(fields, ref_order):
    ps = []
    for i, q in enumerate(fields):
        p = amps.Params.preset(amps.GRAINGROWTH, 0, nx=48 + 16 * i, ny=37, nfields=q, tile=16, seed=7 + i, init_amp=0.3,
                               ref_order=ref_order, mode=amps.END2END_MIX, monitor=amps.MONITOR_RATE, monitor_samples=1,
                               monitor_field=-1, thr_lo=1e-3, thr_hi=5e-2)
        p.dt = ensemble.stable_dt(p.mobil, p.grcoef)
        ps.append(p)
    alone = []
    for p in ps:
        with amps.Simulation(p, init=amps.INIT_SEEDED) as s:
            s.run(25)
            alone.append((s.fields(), s.tiers()))
    sims = [amps.Simulation(p, init=amps.INIT_SEEDED) for p in ps]
    with amps.Ensemble(sims) as ens:
        ens.run(25)
        ens.synchronize()
        for s, (f, t) in zip(sims, alone):
            assert np.array_equal(s.fields(), f)
            assert np.array_equal(s.tiers(), t)
    for s in sims:
        s.close()
