"""Grain growth's step kernels with and without the FP64 code: runs that hold
half or FP32 data only take kernels without it, adaptive runs whose tiles all
stay at half or FP32 those with it -- the same per-tile code, so the same bits.
And ensembles of 16^2 tiles whose members' shared memory does not grow with
their fields (12 fields stage more than 13)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


@pytest.mark.parametrize("nx,ny,tile,q,ref_order,half_arith", [
    (64, 96, 32, 8, 0, 0), (64, 96, 32, 3, 1, 0), (64, 48, 16, 2, 1, 0), (48, 48, 16, 13, 0, 0), (75, 61, 32, 4, 0, 0),
    (75, 61, 16, 12, 1, 0), (64, 96, 32, 2, 1, 1), (64, 48, 16, 2, 0, 2)])
@pytest.mark.parametrize("tier", ["half", "fp32"])
def test_same_bits_without_fp64_code(nx, ny, tile, q, ref_order, half_arith, tier):
    w = amps()
    if tier == "fp32" and half_arith:
        pytest.skip("binary16 arithmetic is half tiles'")
    p = w.Params.preset(w.GRAINGROWTH, 0, nx=nx, ny=ny, nfields=q, tile=tile, ref_order=ref_order, half_arith=half_arith,
                        monitor=w.MONITOR_SPA, monitor_samples=1, monitor_field=-1)
    f = np.random.default_rng(6).random((q, ny, nx)).astype(np.float16).astype(np.float64)
    if tier == "half":
        pure, mixed = dict(mode=w.PURELOW), dict(mode=w.END2END_MIX, thr_lo=1e300, thr_hi=1e300)
        want = w.TIER_HALF
    else:
        pure, mixed = dict(mode=w.PUREHIGH, high_tier=w.TIER_FP32), dict(mode=w.END2END_MIX, thr_lo=-1.0, thr_hi=1e300)
        want = w.TIER_FP32
    out = []
    for kw in (pure, mixed):
        with w.Simulation(p.replace(**kw)) as s:
            s.set_fields(f)
            s.run(13)
            assert np.all(s.tiers() == want)
            out.append(s.fields())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("fields", [(20, 12), (13, 12), (16, 3, 12)])
def test_ensemble_members_that_stage_more_with_fewer_fields(fields):
    w = amps()
    from w3914777_gb300 import ensemble
    ps = []
    for i, q in enumerate(fields):
        p = w.Params.preset(w.GRAINGROWTH, 0, nx=48 + 16 * i, ny=37, nfields=q, tile=16, seed=7 + i, init_amp=0.3,
                            mode=w.END2END_MIX, monitor=w.MONITOR_RATE, monitor_samples=1, monitor_field=-1, thr_lo=1e-3,
                            thr_hi=5e-2)
        p.dt = ensemble.stable_dt(p.mobil, p.grcoef)
        ps.append(p)
    alone = []
    for p in ps:
        with w.Simulation(p, init=w.INIT_SEEDED) as s:
            s.run(25)
            alone.append(s.fields())
    sims = [w.Simulation(p, init=w.INIT_SEEDED) for p in ps]
    with w.Ensemble(sims) as ens:
        ens.run(25)
        ens.synchronize()
        for s, f in zip(sims, alone):
            assert np.array_equal(s.fields(), f)
    for s in sims:
        s.close()
