"""The one-step forward and adjoint kernels at the edges of their ranges:
grids below, at and just past a tile, sides that are not multiples of four
(unaligned rows), both boundaries and stencils, field counts for every split
of fields over warps, unaligned state pointers, even, odd and fractional
anisotropy -- against torch.autograd of the plain float64 restatement."""
import pytest
import torch

import adjoint_ref as ar

pytestmark = pytest.mark.gpu


def amps():
    from w3914777_gb300 import amps as w
    return w


def _check(p, state, dtype, tol_f, tol_g, offset=0, tol_p=None):
    """One step: outputs, input cotangents and parameter gradients, relative to
    the largest reference value."""
    from w3914777_gb300 import adjoint
    w = amps()
    names = adjoint.PARAM_NAMES[p.model]
    ref = state.to(dtype).double().requires_grad_(True)
    v = [torch.tensor(getattr(p, n), dtype=torch.float64, requires_grad=True) for n in names]
    out = ar.kob_step(ref, p, *v, 3) if p.model == w.KOBAYASHI else ar.gg_step(ref, p, *v)
    gen = torch.Generator().manual_seed(4)
    g = torch.randn(state.shape, generator=gen, dtype=torch.float64).to(dtype)
    out.backward(g.double())

    def dev(t):  # on the device, `offset` elements past an aligned address
        buf = torch.zeros(t.numel() + offset, dtype=dtype, device="cuda")
        d = buf[offset:].view(t.shape)
        d.copy_(t)
        return d
    st = adjoint.Stepper(p, dtype=dtype)
    x, go, o, gi = dev(state.to(dtype)), dev(g), dev(torch.zeros_like(state)), dev(torch.zeros_like(state))
    gp = torch.zeros(3, dtype=torch.float64, device="cuda")
    st.forward(x, 3, out=o)
    st.adjoint(x, go, 3, gp, grad_in=gi)
    rel = lambda a, b: float((a.double().cpu() - b).abs().max() / b.abs().max())
    ef, eg = rel(o, out.detach()), rel(gi, ref.grad)
    want = torch.stack([t.grad for t in v])
    ep = rel(gp, want)
    print(f"{tuple(state.shape)} {dtype}: out {ef:.1e} grad {eg:.1e} params {ep:.1e}")
    assert ef <= tol_f and eg <= tol_g
    if tol_p is None:
        assert ep <= tol_g
        return
    # the sums' terms have the random signs of g: their error is relative to the terms' magnitudes
    for k in range(3):
        d = [torch.zeros((), dtype=torch.float64) for _ in range(3)]
        d[k] = torch.ones((), dtype=torch.float64)
        fn = lambda *u: ar.gg_step(ref.detach(), p, *u)
        _, j = torch.func.jvp(fn, tuple(t.detach() for t in v), tuple(d))
        assert float((gp[k].cpu() - want[k]).abs()) <= tol_p * float((j * g.double()).abs().sum())


GG = [(5, 5, 1, 0, 0, 0), (31, 17, 3, 1, 0, 0), (33, 15, 4, 0, 1, 0), (64, 32, 8, 1, 1, 0), (66, 34, 9, 0, 0, 1),
      (36, 40, 5, 1, 0, 1), (100, 7, 32, 1, 1, 0), (640, 250, 2, 1, 0, 0), (604, 300, 6, 0, 0, 0), (320, 420, 8, 1, 0, 3)]


@pytest.mark.parametrize("nx,ny,q,bc,stencil,offset", GG)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_grain_growth_step(nx, ny, q, bc, stencil, offset, dtype):
    """FP64 to 1e-11; FP32 to 40 roundings of the largest term, 40 * 2^-24 <
    3e-6; the parameter sums to 24 * 2^-24 of their terms' magnitudes (about ten
    roundings a term, and at most 64 additions a thread of values whose signs
    keep the partial sums near an eighth of those)."""
    w = amps()
    p = w.Params.preset("graingrowth", 0, nx=nx, ny=ny, nfields=q, bc=bc, stencil=stencil, mode="purehigh", dx=0.9,
                        dy=0.9, gamma=1.3)
    f = torch.rand((q, ny, nx), generator=torch.Generator().manual_seed(nx), dtype=torch.float64)
    d = dtype == torch.float64
    _check(p, f, dtype, 1e-11 if d else 3e-6, 1e-11 if d else 3e-6, offset, None if d else 24 * 2.0 ** -24)


KOB = [(5, 6, 0, 6.0, 0), (32, 8, 1, 6.0, 0), (33, 9, 1, 4.0, 1), (47, 31, 0, 5.0, 0), (64, 64, 1, 2.5, 0),
       (320, 500, 1, 6.0, 3), (353, 481, 0, 16.0, 0)]


@pytest.mark.parametrize("nx,ny,bc,aniso,offset", KOB)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_kobayashi_step(nx, ny, bc, aniso, offset, dtype):
    """A ramp with noise keeps grad phi away from zero, where the angle has no
    derivative.  FP64 to 1e-10 (the bar of the other adjoint tests); FP32 to
    2e-4: the angle's cotangent divides by |grad phi| (differences of 0.02 of
    values near 1, each rounded to 2^-24: 1e-5 relative) and is scaled by the
    anisotropy mode."""
    w = amps()
    p = w.Params.preset("kobayashi", 0, nx=nx, ny=ny, bc=bc, mode="purehigh", aniso=aniso, noise=0.01, seed=9)
    y, x = torch.meshgrid(torch.arange(ny, dtype=torch.float64), torch.arange(nx, dtype=torch.float64), indexing="ij")
    gen = torch.Generator().manual_seed(nx)
    ramp = 0.03 * x + 0.02 * y
    phi = 0.1 + 0.8 * torch.abs(torch.remainder(ramp / 0.8, 2) - 1) if bc else 0.5 + 0.3 * torch.sin(
        2 * torch.pi * (x / nx + y / ny)) + 0.02 * torch.rand(ny, nx, generator=gen, dtype=torch.float64)
    phi = phi + 0.002 * torch.rand(ny, nx, generator=gen, dtype=torch.float64)
    T = 0.4 * torch.rand(ny, nx, generator=gen, dtype=torch.float64)
    d = dtype == torch.float64
    _check(p, torch.stack([phi, T]), dtype, 1e-11 if d else 3e-6, 1e-10 if d else 2e-4, offset)
