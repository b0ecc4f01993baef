"""Grain growth's FP64 tiles: the band kernel of all-FP64 steps and the FP64
tiles of the fused step, at the edges of their ranges (field counts below,
at and off multiples of the warps, one tile, 16^2 and 32^2 tiles, both
stencils, divisors that are a power of two, known and general)."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


@pytest.mark.parametrize("nx,ny,q,tile,stencil,bc,ref_order,dx", [
    (32, 32, 1, 32, 0, 0, 0, 1.0), (96, 64, 3, 32, 0, 1, 0, 0.7), (64, 64, 8, 32, 0, 0, 0, 1.0),
    (64, 33, 17, 32, 0, 0, 0, 0.9), (75, 64, 6, 32, 1, 1, 0, 1.0), (48, 16, 2, 16, 0, 0, 0, 0.5),
    (37, 52, 5, 16, 0, 1, 0, 1.0), (64, 32, 18, 16, 1, 0, 0, 1.0), (16, 16, 1, 16, 0, 1, 1, 0.5),
    (48, 32, 2, 16, 0, 0, 1, 0.5), (50, 64, 3, 32, 0, 1, 1, 0.7), (64, 64, 9, 32, 1, 0, 1, 0.9),
    (32, 48, 20, 16, 0, 0, 1, 1.3)])
def test_plain_fp64_vs_oracle(nx, ny, q, tile, stencil, bc, ref_order, dx):
    """30 plain FP64 steps against the oracle, relative: 1e-13.  A step rounds
    each cell a few times (2^-53 each) and the update, with dt*L*(kappa/dx^2*12
    + 3) < 2, does not amplify; 30 steps stay below 30 * 8 * 2^-53 < 3e-14."""
    w = amps()
    p = w.Params.preset("graingrowth", 0, mode="purehigh", nx=nx, ny=ny, nfields=q, tile=tile, bc=bc, stencil=stencil,
                        ref_order=ref_order, dx=dx, dy=dx, dt=0.02, init_amp=0.5, seed=11 + q)
    f0 = w.init_host(p, w.INIT_SEEDED)
    with w.Simulation(p, init=w.INIT_SEEDED) as s:
        s.run(30)
        f = s.fields()
    o = ob.gg_run(ob.gg_params(nx, ny, q=q, bc=bc, stencil=stencil, dx=dx, dy=dx, dt=0.02, mobil=p.mobil,
                               grcoef=p.grcoef, gamma=p.gamma), list(f0), 30)
    e = max(np.max(np.abs(f[k] - o[k])) for k in range(q)) / max(np.max(np.abs(v)) for v in o)
    print(f"{nx}x{ny} q {q} tile {tile} ref {ref_order}: {e:.2e}")
    assert e <= 1e-13


@pytest.mark.parametrize("nx,ny,q,tile,ref_order", [(96, 64, 3, 32, 0), (64, 64, 8, 32, 1), (77, 50, 12, 32, 0),
                                                    (64, 48, 2, 16, 1), (33, 48, 17, 16, 0)])
def test_fused_fp64_tiles_are_the_band_kernels_bits(nx, ny, q, tile, ref_order):
    """A schedule that holds every tile at FP64 runs the fused step's FP64
    tiles; plain FP64 the band kernel: the same bits."""
    w = amps()
    p = w.Params.preset("graingrowth", 0, nx=nx, ny=ny, nfields=q, tile=tile, ref_order=ref_order, bc=1, init_amp=0.5,
                        monitor=w.MONITOR_RATE, thr_lo=1e-5, thr_hi=1e-2)
    with w.Simulation(p.replace(mode="purehigh"), init=w.INIT_SEEDED) as s:
        s.run(25)
        a = s.fields()
    with w.Simulation(p) as s:
        s.set_tier_schedule(np.full((1,) + s.ntiles, w.TIER_FP64, dtype=np.uint8))
        s.init(w.INIT_SEEDED)
        s.run(25)
        b = s.fields()
    assert np.array_equal(a, b)


@pytest.mark.parametrize("monitor", [1, 2, 3])
@pytest.mark.parametrize("samples", [0, 1])
def test_fp64_monitor_metric(monitor, samples):
    """The metric of the all-FP64 first period's monitor step, from its fields
    before and after (the range, or the last step's or the period's change):
    equal bit for bit (maxima of exactly formed differences)."""
    w = amps()
    nx, ny, q, T = 75, 64, 3, 32
    p = w.Params.preset("graingrowth", 0, mode="end2end_mix", nx=nx, ny=ny, nfields=q, tile=T, bc=1, init_amp=0.5,
                        monitor=monitor, monitor_samples=samples, thr_lo=0.0, thr_hi=0.0)
    with w.Simulation(p, init=w.INIT_SEEDED) as s:
        first = s.fields()
        s.run(9)
        before = s.fields()
        s.run(1)
        after, got = s.fields(), s.metric()
    if monitor == 1:
        at = [0, 10, 21, 31]
    else:
        at = [4, 12, 20, 28]
    want = np.zeros_like(got)
    for ty in range(got.shape[0]):
        for tx in range(got.shape[1]):
            ys, xs = (range(T), range(T)) if samples else (at, at)
            idx = np.ix_(range(q), [ty * T + y for y in ys if ty * T + y < ny], [tx * T + x for x in xs if tx * T + x < nx])
            v = after[idx]
            if v.size == 0:
                continue
            if monitor == 1:
                lo, hi = v.min((1, 2)), v.max((1, 2))
                m = (hi - lo).max() if samples else (np.maximum(hi, 0.0) - np.minimum(lo, 1.0)).max()
            elif monitor == 2:
                m = np.abs(v - first[idx]).max()
            else:
                m = float(np.abs(v.astype(np.float32) - before[idx].astype(np.float32)).max()) * p.cadence
            want[ty, tx] = m
    assert np.array_equal(got, want)
