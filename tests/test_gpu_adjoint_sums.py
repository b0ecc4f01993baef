"""The FP32 adjoint's parameter sums across a block are formed with no less than
double precision and range.  A uniform state of eight fields of 1/4 with
gamma = 1.5 makes every cell's term an exact multiple of its cotangent
(e*b = 3/32, e*(S - e^2) = 7/64), and each warp advances one field, so the sums
over the fields are exact in double: what they must give is known to the bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sums(g):
    """dL/d(L, gamma) / (-dt) and / (-2 dt L) of one step, field f's cotangent g[f] everywhere."""
    from w3914777_gb300 import adjoint
    from w3914777_gb300 import amps as w
    p = w.Params.preset(w.GRAINGROWTH, 0, nx=64, ny=32, nfields=8, gamma=1.5, mobil=1.0, dt=2.0 ** -5)
    x = torch.full((8, p.ny, p.nx), 0.25, dtype=torch.float32, device="cuda")
    go = torch.tensor(g, dtype=torch.float32, device="cuda")[:, None, None].expand_as(x).contiguous()
    gp = torch.zeros(3, dtype=torch.float64, device="cuda")
    adjoint.Stepper(p, dtype=torch.float32).adjoint(x, go, 0, gp)
    gp = gp.cpu()
    return float(gp[0]) / -p.dt, float(gp[2]) / (-2.0 * p.dt * p.mobil), p.nx * p.ny


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 60, 2.0 ** -60])
@pytest.mark.parametrize("g", [
    (1.0, 2.0 ** -25, 2.0 ** -51, -1.0, -(2.0 ** -25), 0.0, 0.0, 0.0),
    (2.0 ** -51, 1.0, -(2.0 ** -25), 2.0 ** -25, -1.0, 0.0, 0.0, 2.0 ** -52),
])
def test_sums_keep_what_double_keeps(g, scale):
    gl, gg, n = _sums([v * scale for v in g])
    want = sum(g) * scale  # exact in double in this order
    assert want != 0.0
    assert gl == n * want * 3 / 32
    assert gg == n * want * 7 / 64


def test_sums_past_the_range_of_float():
    g = 2.0 ** 126  # eight cells a thread: 3/4 and 7/8 of it; eight warps: past 2^128
    gl, gg, n = _sums([g] * 8)
    assert gl == n * 8 * g * 3 / 32
    assert gg == n * 8 * g * 7 / 64
