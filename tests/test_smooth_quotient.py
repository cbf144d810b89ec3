"""The smooth union's quotient gap / k from the reciprocal of its one width k
(smooth_min_by): two corrections by the remainder give IEEE's quotient for
every gap the formula divides, widths from 2^-60 to 2^60, mantissas of all
ones and powers of two among them.  The device's two fused operations are
restated exactly in float64, and in rationals where that could round twice."""
from fractions import Fraction

import numpy as np
import pytest

f32, f64 = np.float32, np.float64


def _round32(x):
    """A rational to the nearest float32 (ties to even)."""
    if x == 0:
        return f32(0)
    e = 0
    m = abs(x)
    while m >= 2 ** 24:
        m /= 2
        e += 1
    while m < 2 ** 23:
        m *= 2
        e -= 1
    n, r = divmod(m.numerator, m.denominator)
    half = Fraction(r, m.denominator)
    n += half > Fraction(1, 2) or (half == Fraction(1, 2) and n & 1)
    return f32(np.ldexp(f64(n), e) * (1 if x > 0 else -1))


def _fma(a, b, c):
    return _round32(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)))


def _exact(gap, k, rk):
    h = f32(gap * rk)
    for _ in range(2):
        h = _fma(_fma(-k, h, gap), rk, h)
    return h


def _gaps(k, rng, n):
    """Differences k - |a - b| of float32 numbers, from a rounding unit of k up to k."""
    t = np.concatenate([rng.uniform(0, 1, n // 2), 1 - 2.0 ** rng.uniform(-24, 0, n // 2)]).astype(f32)
    g = (k - (k * t).astype(f32)).astype(f32)
    return g[g > 0]


@pytest.mark.parametrize("seed", range(4))
def test_quotient_is_ieee(seed):
    rng = np.random.default_rng(seed)
    widths = [f32(0.05), f32(1.0), f32(2.0 ** -60), f32(2.0 ** 60), np.nextafter(f32(2), f32(0)), np.nextafter(f32(1), f32(0)),
              np.nextafter(f32(1), f32(2))]
    widths += list((rng.uniform(1, 2, 60) * 2.0 ** rng.integers(-59, 59, 60)).astype(f32))
    for k in widths:
        rk = f32(1) / k
        gap = _gaps(k, rng, 4000)
        want = gap / k
        h = gap * rk
        for _ in range(2):
            r = (gap.astype(f64) - f64(k) * h.astype(f64)).astype(f32)
            h = (h.astype(f64) + r.astype(f64) * f64(rk)).astype(f32)
        for i in np.nonzero(h != want)[0]:
            h[i] = _exact(gap[i], k, rk)
        assert np.array_equal(h, want), k
        for i in rng.integers(0, len(gap), 3):  # the float64 restatement itself
            assert _exact(gap[i], k, rk) == want[i]
