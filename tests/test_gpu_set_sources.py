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


def _managed(nbytes):
    """Managed memory, from the driver."""
    cuda = ctypes.CDLL("libcuda.so.1")
    p = ctypes.c_uint64()
    assert cuda.cuMemAllocManaged(ctypes.byref(p), ctypes.c_size_t(nbytes), 1) == 0
    return cuda, p


@pytest.mark.parametrize("run", ["plain", "spa", "rate"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("source", ["bytes", "managed", "inside"])
def test_device_sources_that_a_kernel_cannot_or_may_read_in_place(run, dtype, source):
    """A device array at an odd address, and managed memory, are copied; one
    that ends with its allocation is read in place."""
    tt, code, npt = (torch.float64, w.F64, np.float64) if dtype == "f64" else (torch.float32, w.F32, np.float32)
    want = _values((3, NY, NX), 7)
    host = np.ascontiguousarray(want.numpy().astype(npt))
    cuda = p = None
    if source == "managed":
        torch.cuda.synchronize()
        cuda, p = _managed(host.nbytes)
        ctypes.memmove(p.value, host.ctypes.data, host.nbytes)
        ptr = p.value
    elif source == "bytes":
        buf = torch.zeros(host.nbytes + 16, dtype=torch.uint8, device="cuda")
        buf[2:2 + host.nbytes].copy_(torch.from_numpy(host.view(np.uint8).reshape(-1)))
        ptr = buf.data_ptr() + 2
    else:
        buf = torch.zeros(host.size + 64, dtype=tt, device="cuda")
        buf[64:].copy_(torch.from_numpy(host).reshape(-1))
        ptr = buf[64:].data_ptr()
    torch.cuda.synchronize()
    with _sim(run) as s:
        _set(s, None, ptr, code, 1)
        got = s.fields()
    if p is not None:
        cuda.cuMemFree_v2(p)
    assert np.array_equal(got, want.numpy())
