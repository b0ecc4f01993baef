"""What amps_set_field(s) may assume about the caller's array: it has been read
when the call returns, whatever the mode, the monitor and the kind of source."""
import ctypes

import numpy as np
import pytest
import torch

from w3914777_gb300 import amps as w

pytestmark = pytest.mark.gpu

NX, NY = 512, 384
RUNS = {"plain": dict(mode="purehigh"), "fp32": dict(mode="purehigh", high_tier=w.TIER_FP32),
        "low": dict(mode="purelow"), "gram": dict(mode="gram1", gram_ratio=0.5),
        "spa": dict(mode="end2end_mix", monitor=w.MONITOR_SPA, monitor_samples=1, thr_lo=0.0, thr_hi=0.0),
        "tem": dict(mode="end2end_mix", monitor=w.MONITOR_TEM, thr_lo=1e-4, thr_hi=1e-4),
        "rate": dict(mode="end2end_mix", monitor=w.MONITOR_RATE, thr_lo=1e-4, thr_hi=1e-4)}


def _sim(run, nfields=3):
    return w.Simulation(w.Params.preset("graingrowth", 0, nx=NX, ny=NY, nfields=nfields, **RUNS[run]), init=w.INIT_SEEDED)


def _set(s, field, ptr, dtype, on_device):
    if field is None:
        rc = w.lib().amps_set_fields(s.h, ctypes.c_void_p(ptr), dtype, on_device)
    else:
        rc = w.lib().amps_set_field(s.h, field, ctypes.c_void_p(ptr), dtype, on_device)
    assert rc == 0


# multiples of 1/1024 up to 1: every tier stores them exactly
def _values(shape, seed):
    return torch.from_numpy(np.random.default_rng(seed).integers(0, 1025, shape) / 1024.0)


@pytest.mark.parametrize("run", sorted(RUNS))
@pytest.mark.parametrize("field", [None, 1])
@pytest.mark.parametrize("source", ["device", "pinned", "pageable"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_source_may_be_overwritten_on_return(run, field, source, dtype):
    """The stream is busy with a run when the state is set; the source is
    overwritten as soon as the call returns."""
    tt, code = (torch.float64, w.F64) if dtype == "f64" else (torch.float32, w.F32)
    shape = (3, NY, NX) if field is None else (NY, NX)
    want = _values(shape, 5)
    src = want.to(tt).clone()
    if source == "device":
        src = src.cuda()
    elif source == "pinned":
        src = src.pin_memory()
    with _sim(run) as s:
        s.synchronize()
        torch.cuda.synchronize()
        s.run(300)
        _set(s, field, src.data_ptr(), code, int(source == "device"))
        src.fill_(0.5)
        torch.cuda.synchronize()
        got = s.fields()
    assert np.array_equal(got if field is None else got[field], want.numpy())


@pytest.mark.parametrize("run", sorted(RUNS))
@pytest.mark.parametrize("field", [None, 1])
def test_float_device_source_follows_the_default_stream(run, field):
    """A float array that work on the default stream is still to write when the
    state is set, with no synchronisation of the caller's."""
    shape = (3, NY, NX) if field is None else (NY, NX)
    want = _values(shape, 6)
    made = want.float().cuda()
    src = torch.full(shape, 0.5, dtype=torch.float32, device="cuda")
    with _sim(run) as s:
        s.synchronize()
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)
        src.copy_(made)
        _set(s, field, src.data_ptr(), w.F32, 1)
        got = s.fields()
    assert np.array_equal(got if field is None else got[field], want.numpy())
