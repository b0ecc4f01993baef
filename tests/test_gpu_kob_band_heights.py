"""Kobayashi's FP64 tiles in adaptive runs: however many there are, and so
whatever the height of their bands and the bands a CTA loops over, a run whose
tiles are all at FP64 has a plain run's bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


# tiles: 40, 80, 256 of 32^2 (bands of 4, 8, 16 rows); 144, 256, 512 of 16^2 (8, 16, 16)
@pytest.mark.parametrize("nx,ny,tile,ref_order,bc", [
    (256, 160, 32, 0, 1), (320, 256, 32, 1, 0), (512, 512, 32, 0, 0), (192, 192, 16, 0, 0), (256, 256, 16, 1, 1),
    (512, 256, 16, 0, 1)])
def test_adaptive_bands_are_the_plain_runs_bits(nx, ny, tile, ref_order, bc):
    w = amps()
    p = w.Params.preset("kobayashi", 2, nx=nx, ny=ny, tile=tile, ref_order=ref_order, bc=bc, noise=0.01, seed=5,
                        monitor=w.MONITOR_SPA, monitor_samples=1, thr_lo=-1.0, thr_hi=-1.0)
    with w.Simulation(p.replace(mode=w.PUREHIGH), init=w.INIT_REFERENCE) as s:
        s.run(12)
        a = s.fields()
    with w.Simulation(p.replace(mode=w.END2END_MIX), init=w.INIT_REFERENCE) as s:
        s.run(12)
        b = s.fields()
        assert np.all(s.tiers() == w.TIER_FP64)
    assert np.array_equal(a, b)
