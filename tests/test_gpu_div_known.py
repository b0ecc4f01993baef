"""The reference-order FP64 tiles divide by the known dx*dy with a product and a
correction where the divisor allows it: the quotient is IEEE division's, to the
bit, for divisors of each kind and numerators of every exponent.

A grain-growth step with L = kappa = dt = 1 from a field that is zero but for
isolated cells leaves s / (dx*dy) in the zero cells, s their only neighbour."""
import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kind(d):
    """0: the general division; 1: a power of two; 2: product and correction."""
    m, ex = math.frexp(d)
    if ex < -63 or ex > 64:
        return 0
    if m == 0.5:
        return 1
    return 2 if abs(1 - Fraction(d) * Fraction(1.0 / d)) <= Fraction(1, 2 ** 54) else 0


def _divisors():
    rng = np.random.default_rng(11)
    ds = [0.25, 1.0, 2.0 ** 20, 2.0 ** -40, 2.0 ** 70, 2.0 ** -70, 0.03 * 0.03, 0.5 * 0.3, 1.0 / 3.0, 1.0 + 2.0 ** -52,
          2.0 - 2.0 ** -52, 1e-25, 1e25]
    ds += [float(v) for v in np.ldexp(1.0 + rng.random(19), rng.integers(-60, 60, 19))]
    assert {_kind(d) for d in ds} == {0, 1, 2}
    return ds


def _numerators(n):
    rng = np.random.default_rng(12)
    x = np.ldexp(1.0 + rng.random(n), rng.integers(-1074, 1024, n)) * rng.choice([-1.0, 1.0], n)
    x[:12] = [0.0, 5e-324, -5e-324, 2.0 ** -1022, 2.0 ** -895, 2.0 ** -896, 2.0 ** 897, 2.0 ** 898, -2.0 ** 1023,
              np.finfo(float).max, np.inf, -np.inf]
    x[12] = np.nan
    x[13:200] = np.ldexp(1.0 + rng.random(187), rng.integers(-60, 60, 187))
    return x


@pytest.mark.parametrize("stencil", [0, 1])
def test_quotients_are_ieee(stencil):
    from w3914777_gb300 import amps as w
    side = 96
    x = _numerators((side // 3) ** 2).reshape(side // 3, side // 3)
    f = np.zeros((2, side, side))
    f[0, 1::3, 1::3] = x
    for d in _divisors():
        p = w.Params.preset(w.GRAINGROWTH, 1, nx=side, ny=side, nfields=2, mode=w.PUREHIGH, ref_order=1, tile=32,
                            stencil=stencil, dx=d, dy=1.0, dt=1.0, mobil=1.0, grcoef=1.0)
        with w.Simulation(p) as s:
            s.set_fields(f)
            s.run(1)
            got = s.field(0)[1::3, 2::3]
        with np.errstate(over="ignore", under="ignore"):
            want = x / d
        assert np.array_equal(got, want, equal_nan=True), d
