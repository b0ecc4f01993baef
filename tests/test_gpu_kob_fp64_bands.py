"""Kobayashi's FP64 tiles in row bands, at the edges of their range: one tile,
few tiles (bands of 4 rows), many (bands of 8 and 16), 16^2 and 32^2 tiles,
both boundaries, the reference's order and the library's, cell sizes whose
divisions are exact, known and general."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


@pytest.mark.parametrize("nx,ny,tile,bc,ref_order,dx,dy", [
    (32, 32, 32, 0, 1, 0.03, 0.03), (16, 16, 16, 1, 1, 0.03, 0.03), (96, 64, 32, 1, 1, 0.03, 0.04),
    (128, 96, 32, 1, 0, 0.03, 0.03), (48, 80, 16, 0, 0, 0.03, 0.03), (64, 64, 32, 0, 1, 0.03125, 0.03125),
    (64, 64, 16, 1, 1, 0.035, 0.029), (512, 512, 32, 1, 1, 0.03, 0.03), (640, 512, 16, 0, 1, 0.03, 0.03)])
def test_plain_fp64_vs_oracle(nx, ny, tile, bc, ref_order, dx, dy):
    """8 steps of a noisy dendrite against the oracle, to 1e-12 relative (the
    bar of the other parity tests: the device's atan2, cos, sin and atan are
    within an ulp or two of glibc's, and a few steps do not amplify that)."""
    w = amps()
    p = w.Params.preset("kobayashi", 2, mode="purehigh", nx=nx, ny=ny, tile=tile, bc=bc, ref_order=ref_order, dx=dx,
                        dy=dy, init_offset=0, init_r2=30.0, noise=0.01, seed=5)
    rng = np.random.default_rng(3)
    f0 = w.init_host(p, w.INIT_REFERENCE)
    f0[0] = np.clip(f0[0] + 0.02 * rng.random(f0[0].shape), 0, 1.02)
    with w.Simulation(p) as s:
        s.set_fields(f0)
        s.run(8)
        f = s.fields()
    o = ob.kob_run(ob.kob_params(nx, ny, bc=bc, dx=dx, dy=dy, noise=0.01, seed=5), f0[0], f0[1], 8)
    e = max(np.max(np.abs(f[k] - o[k])) for k in range(2)) / max(np.max(np.abs(o[0])), 1.0)
    print(f"{nx}x{ny} tile {tile} bc {bc} ref {ref_order}: {e:.2e}")
    assert e <= 1e-12


def test_bands_are_the_whole_tiles_bits():
    """An adaptive run whose tiles all stay at FP64 takes whole tiles on its
    monitor steps and bands (looped over by one CTA an SM) on the others; a
    plain run bands only: the same bits."""
    w = amps()
    for nx, ny, tile, ref in ((192, 160, 32, 1), (64, 48, 16, 0)):
        p = w.Params.preset("kobayashi", 2, nx=nx, ny=ny, tile=tile, ref_order=ref, noise=0.01, seed=5, bc=1,
                            monitor=w.MONITOR_SPA, monitor_samples=1, thr_lo=-1.0, thr_hi=-1.0)
        with w.Simulation(p.replace(mode=w.PUREHIGH), init=w.INIT_REFERENCE) as s:
            s.run(30)
            a = s.fields()
        with w.Simulation(p.replace(mode=w.END2END_MIX), init=w.INIT_REFERENCE) as s:
            s.run(30)
            b = s.fields()
            assert np.all(s.tiers() == w.TIER_FP64)
        assert np.array_equal(a, b)
