"""Setting and reading the state: every tier and mixtures of them, both tiles,
odd and ragged sides, double and float arrays on the host and on the device,
unaligned device arrays; large tile maps (several tiles a thread in the
classification)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


def _stored(f, tiers, tile):
    """What storing f at each tile's tier keeps."""
    out = f.copy()
    for ty in range(tiers.shape[0]):
        for tx in range(tiers.shape[1]):
            s = np.s_[:, ty * tile:(ty + 1) * tile, tx * tile:(tx + 1) * tile]
            if tiers[ty, tx] == 0:
                out[s] = f[s].astype(np.float32).astype(np.float16)
            elif tiers[ty, tx] == 1:
                out[s] = f[s].astype(np.float32)
    return out


@pytest.mark.parametrize("nx,ny,q,tile", [(32, 32, 1, 32), (33, 47, 5, 32), (100, 64, 4, 32), (16, 50, 3, 16),
                                          (61, 33, 9, 16), (128, 96, 8, 16)])
@pytest.mark.parametrize("mode", ["purehigh", "fp32", "purelow", "gram"])
@pytest.mark.parametrize("offset", [0, 1])
def test_round_trip(nx, ny, q, tile, mode, offset):
    w = amps()
    p = w.Params.preset("graingrowth", 0, nx=nx, ny=ny, nfields=q, tile=tile, mode="purehigh")
    if mode == "fp32":
        p.high_tier = w.TIER_FP32
    elif mode == "purelow":
        p.mode = w.PURELOW
    elif mode == "gram":
        p = p.replace(mode="gram1", gram_ratio=0.5)
    f = np.random.default_rng(nx + q).uniform(-1, 1, (q, ny, nx))
    with w.Simulation(p) as s:
        tiers = s.tiers()
        if mode == "gram":
            s.set_fields(f)
            tiers = s.tiers()
        for dtype, code, tt in ((np.float64, w.F64, torch.float64), (np.float32, w.F32, torch.float32)):
            g = f.astype(dtype)
            want = _stored(g.astype(np.float64), tiers, tile)
            buf = torch.zeros(g.size + offset, dtype=tt, device="cuda")
            d = buf[offset:].view(g.shape)
            d.copy_(torch.from_numpy(g))
            torch.cuda.synchronize()
            s.set_fields_device(d.data_ptr(), code)
            d.zero_()  # the state was read before the call returned
            torch.cuda.synchronize()
            assert np.array_equal(s.fields(), want)
            assert np.array_equal(s.fields(np.float32), want.astype(np.float32))
            for out_t, out_c in ((torch.float64, w.F64), (torch.float32, w.F32)):
                o = torch.full((g.size + offset + 1,), 7.0, dtype=out_t, device="cuda")
                torch.cuda.synchronize()
                s.get_fields_device(o[offset:].data_ptr(), out_c)
                assert np.array_equal(o[offset:-1].view(g.shape).cpu().numpy(), want.astype(o.cpu().numpy().dtype))
                assert float(o[-1]) == 7.0 and (offset == 0 or float(o[0]) == 7.0)


@pytest.mark.parametrize("nx,ny,bc", [(32 * 16, 65 * 16, 0), (130 * 16, 33 * 16, 1), (1120 * 16, 16, 0), (300 * 16, 301 * 16, 1)])
def test_large_tile_maps(nx, ny, bc):
    """More tiles than threads: the tier map by thresholds of the spatial metric,
    its counts (through the tile-step statistics) and the run that follows,
    whose launch order visits every tile once."""
    w = amps()
    p = w.Params.preset("graingrowth", 0, nx=nx, ny=ny, nfields=1, tile=16, bc=bc, monitor=w.MONITOR_SPA,
                        monitor_samples=1, thr_lo=0.3, thr_hi=0.6)
    rng = np.random.default_rng(nx)
    amp = np.kron(rng.choice([0.01, 0.2, 0.45], (ny // 16, nx // 16)), np.ones((16, 16)))
    f = (amp * rng.uniform(-1, 1, (ny, nx)))[None]
    with w.Simulation(p) as s, w.Simulation(p.replace(mode="purehigh")) as plain:
        s.set_fields(f)
        m = s.measure_tiles()
        mm = m.copy()
        mm[1:] = np.maximum(mm[1:], m[:-1])
        mm[:-1] = np.maximum(mm[:-1], m[1:])
        mm[:, 1:] = np.maximum(mm[:, 1:], m[:, :-1])
        mm[:, :-1] = np.maximum(mm[:, :-1], m[:, 1:])
        want = np.where(mm >= 0.6, 2, np.where(mm >= 0.3, 1, 0))
        assert np.array_equal(s.tiers(), want)
        s.run(10)
        assert s.stats()["tile_steps"] == [10 * int((want == k).sum()) for k in range(3)]
        plain.set_fields(f)
        plain.run(10)
        assert np.abs(s.fields() - plain.fields()).max() <= 0.45 * 10 * 2.0 ** -11  # ten half roundings
