"""Sintering's half/FP32 tiles (32^2: four cells a thread) and FP64 row bands
against the oracle's plain FP64 step at the edges of their ranges: one tile,
one particle, odd and many particles, both boundaries, states with bulk 0/1,
tails, negative zeros and everything in between."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


def _state(n, ny, nx, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:ny, 0:nx]
    f = np.zeros((n + 1, ny, nx))
    for k in range(n):
        cx, cy, r = rng.uniform(0, nx), rng.uniform(0, ny), rng.uniform(6, 12)
        f[k + 1] = 0.5 * (1 - np.tanh((np.hypot(x - cx, y - cy) - r) / 1.5))
    f[f < 1e-6] = 0
    f[f > 1 - 1e-6] = 1
    f[0] = np.clip(f[1:].sum(0), 0, 1)
    f[1, 0, :3] = -0.0
    return f


CASES = [(32, 32, 1, 32, 0), (64, 32, 2, 32, 1), (96, 64, 3, 32, 0), (64, 64, 16, 32, 1), (128, 96, 5, 32, 0),
         (48, 32, 4, 16, 1), (128, 128, 17, 32, 0)]


def _oracle(p, f, steps):
    return ob.sint_run(ob.sint_params(p.nx, p.ny, n=p.nfields, bc=p.bc, dx=p.dx, dy=p.dy, dt=p.dt, coefm=p.coefm,
                                      coefk=p.coefk, coefl=p.coefl, dvol=p.dvol, dvap=p.dvap, dsur=p.dsur,
                                      dgrb=p.dgrb), f[0], list(f[1:]), steps)


@pytest.mark.parametrize("nx,ny,n,tile,bc", CASES)
@pytest.mark.parametrize("kind", ["f64", "bands", "f32"])
def test_one_and_more_steps_vs_oracle(nx, ny, n, tile, bc, kind):
    """FP64 (the band kernel, and bands looped over beside other tiers) to
    1e-12; FP32 tiles beside half ones, one step, to 3e-5: c moves by
    dt*mob*lap(mu), whose FP32 mobility has a relative error of a few 2^-24 and
    whose mu, formed in double from fields rounded to 2^-24, has lap(mu) ~
    2^-24 * 16 * (2A + 8 coefm/dx^2) ~ 2e-4, times dt*mob <= 2e-3."""
    w = amps()
    p = w.Params.preset("sintering", 0, nx=nx, ny=ny, nfields=n, tile=tile, bc=bc, mode="purehigh", ref_order=0)
    f = _state(n, ny, nx, 3 + n)
    steps = 12 if kind == "f64" else 9 if kind == "bands" else 1
    if kind == "f64":
        with w.Simulation(p) as s:
            s.set_fields(f)
            s.run(steps)
            g = s.fields()
    else:
        p = p.replace(mode=w.END2END_MIX, monitor=w.MONITOR_SPA, monitor_samples=1, thr_lo=0.1, thr_hi=0.5)
        with w.Simulation(p) as s:
            tiers = np.full((1,) + s.ntiles, w.TIER_FP64 if kind == "bands" else w.TIER_FP32, dtype=np.uint8)
            s.set_tier_schedule(tiers)
            s.set_fields(f)
            s.run(steps)
            g = s.fields()
    c, etas = _oracle(p, f, steps)
    o = np.stack([c] + list(etas))
    e = np.abs(g - o).max()
    print(f"{nx}x{ny} n {n} tile {tile} bc {bc} {kind}: {e:.2e}")
    assert e <= (3e-5 if kind == "f32" else 1e-12)


@pytest.mark.parametrize("bc", [0, 1])
def test_half_bulk_is_exact(bc):
    """Half tiles of pure bulk (c and every eta 0 or 1, a particle each side of
    a straight boundary outside them) stay as they are, bit for bit."""
    w = amps()
    p = w.Params.preset("sintering", 0, nx=96, ny=96, nfields=3, tile=32, bc=bc, mode="purelow", ref_order=0)
    f = np.zeros((4, 96, 96))
    f[0], f[2] = 1, 1
    with w.Simulation(p) as s:
        s.set_fields(f)
        s.run(20)
        assert np.array_equal(s.fields(), f)
    with w.Simulation(p) as s:
        s.set_fields(0 * f)
        s.run(20)
        assert not s.fields().any()
