"""The diagnostics on the tiered state, at the edges of their range: one tile,
ragged grids, both tiles and boundaries, every tier (and all three at once),
labels below the threshold, grains that wrap, against numpy
-- counts and lengths exact, sums to rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


def _state(q, ny, nx, seed):
    rng = np.random.default_rng(seed)
    f = rng.random((q, ny, nx))
    for _ in range(3):  # blobs a few cells wide, with single-cell specks left in
        f = 0.25 * (f + np.roll(f, 1, 1) + np.roll(f, 1, 2) + np.roll(f, (1, 1), (1, 2)))
    return np.round(2 * f + 0.2 * rng.random((q, ny, nx)), 3)


@pytest.mark.parametrize("nx,ny,q,tile,bc,tiers", [
    (32, 32, 2, 32, 0, "f64"), (16, 16, 3, 16, 0, "f32"), (16, 33, 1, 16, 1, "f32"), (100, 75, 4, 32, 0, "f32"),
    (33, 64, 9, 32, 1, "half"), (97, 50, 5, 16, 0, "half"), (160, 128, 3, 32, 0, "mixed"), (75, 70, 8, 16, 1, "mixed"),
    (640, 515, 32, 32, 0, "f32")])
def test_diagnostics_vs_numpy(nx, ny, q, tile, bc, tiers):
    w = amps()
    p = w.Params.preset("graingrowth", 0, nx=nx, ny=ny, nfields=q, tile=tile, bc=bc, mode="purehigh", dx=0.5, dy=0.7)
    if tiers == "f32":
        p.high_tier = w.TIER_FP32
    elif tiers == "half":
        p.mode = w.PURELOW
    elif tiers == "mixed":
        p = p.replace(mode="gram2", gram_ratio=0.5)
    with w.Simulation(p) as s:
        s.set_fields(_state(q, ny, nx, 5))
        if tiers == "mixed":
            t = np.random.default_rng(1).integers(0, 2, s.ntiles).astype(np.uint8) * 2
            s.set_tiers(t)
        f = s.fields()  # as stored
        for level in (0.9, 1.05, 5.0, -1.0):
            got = s.interface(0, level)
            a = f[0] >= level
            ys, xs = np.nonzero(a)
            ex = (a != np.roll(a, -1, 1)) if bc == 0 else a[:, 1:] != a[:, :-1]
            ey = (a != np.roll(a, -1, 0)) if bc == 0 else a[1:] != a[:-1]
            assert got["cells"] == a.sum()
            assert abs(got["perimeter"] - (ex.sum() * p.dy + ey.sum() * p.dx)) <= 1e-12 * max(1.0, got["perimeter"])
            box = (xs.min(), xs.max(), ys.min(), ys.max()) if len(xs) else (-1,) * 4
            assert (got["xmin"], got["xmax"], got["ymin"], got["ymax"]) == box
        for thr in (0.0, 1.05, 1.25):
            lab = np.where(f.max(0) >= thr, f.argmax(0), -1)
            want = _components(lab, bc)
            got = s.grains(thr)
            assert (got["grains"], got["cells"]) == (want, int((lab >= 0).sum()))
            assert s.grains(thr) == got
        lab = f.argmax(0)
        want = np.zeros((q, q))
        for ax, d in ((1, p.dy), (0, p.dx)):
            a, b = (lab, np.roll(lab, -1, ax)) if bc == 0 else (np.delete(lab, -1, ax), np.delete(lab, 0, ax))
            np.add.at(want, (a[a != b], b[a != b]), d)
        want = want + want.T
        got = s.boundary_lengths()
        assert np.allclose(got, want, rtol=1e-13, atol=0)
        assert np.array_equal(s.boundary_lengths(), got)
        for k in (0, q - 1):
            assert abs(s.reduce(k, w.REDUCE_SUM) - f[k].sum()) <= 1e-14 * nx * ny * 2
            assert s.reduce(k, w.REDUCE_MIN) == f[k].min() and s.reduce(k, w.REDUCE_MAX) == f[k].max()
            assert abs(s.reduce(k, w.REDUCE_SUMSQ) - (f[k] ** 2).sum()) <= 1e-14 * nx * ny * 4
        got = s.measure_tiles(w.MONITOR_SPA)
        for ty in range(got.shape[0]):
            for tx in range(got.shape[1]):
                v = f[:, ty * tile:(ty + 1) * tile, tx * tile:(tx + 1) * tile]
                assert got[ty, tx] == (v.max((1, 2)) - v.min((1, 2))).max()
        s.store_temporal_reference()
        assert not s.measure_tiles(w.MONITOR_TEM).any()


def _components(lab, bc):
    """Connected components of equal non-negative labels, by spreading minima."""
    big = lab.size
    c = np.where(lab >= 0, np.arange(lab.size).reshape(lab.shape), big)
    while True:
        n = c.copy()
        for ax in (0, 1):
            for sh in (1, -1):
                o, m = np.roll(n, sh, ax), np.roll(lab, sh, ax)
                ok = (m == lab) & (lab >= 0)
                if bc:
                    edge = [slice(None)] * 2
                    edge[ax] = 0 if sh == 1 else -1
                    ok[tuple(edge)] = False
                n = np.where(ok, np.minimum(n, o), n)
        flat = np.append(n.ravel(), big)
        n = flat[n]  # pointer jumping
        if np.array_equal(n, c):
            return len(np.unique(c[lab >= 0]))
        c = n
