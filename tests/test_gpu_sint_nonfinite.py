"""Sintering's half and FP32 tiles on states that are not finite: an infinity
is no bulk value, so it must not be taken back to a finite one."""
import numpy as np
import pytest

from w3914777_gb300 import amps as w

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("n", [1, 3])
@pytest.mark.parametrize("tier", ["half", "fp32"])
@pytest.mark.parametrize("where", ["all", "patch", "eta"])
def test_infinite_cells_stay_not_finite(tile, n, tier, where):
    p = w.Params.preset("sintering", 0, nx=64, ny=64, nfields=n, tile=tile, ref_order=0, mode="end2end_mix",
                        monitor=w.MONITOR_SPA, monitor_samples=1, thr_lo=0.1, thr_hi=0.5)
    f = np.zeros((n + 1, 64, 64))
    at = np.s_[:, :] if where == "all" else np.s_[8:13, 20:27]
    if where != "eta":
        f[0][at] = np.inf
    f[1][at] = np.inf
    with w.Simulation(p) as s:
        s.set_tier_schedule(np.full((1,) + s.ntiles, w.TIER_HALF if tier == "half" else w.TIER_FP32, dtype=np.uint8))
        s.set_fields(f)
        s.run(1)
        g = s.fields()
    assert not np.isfinite(g[0][at]).any()
