"""The reciprocal of a pivot in the FP64 elimination (recip64): the hardware's
approximation and one third-order step where neither can overflow or lose bits
(exponent fields 64 to 1983), the division elsewhere.  A system of uncoupled
diagonal blocks and a right-hand side of ones returns it as it is: blocks of one
species (a CTA by itself, and in one launch) and of 32 (a cluster).

Bound: the approximation sees and keeps 20 bits of the significand, so e = 1 - a x
is at most 2^-19 besides its own error; x (1 + e + e^2) leaves e^3 = 2^-57 of the result,
at most 1/16 ulp, and rounds once: 0.57 ulp.  The division's results are exact."""
from fractions import Fraction

import numpy as np
import pytest

from test_noalloc_shapes import _call

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _values(n, lo, hi, seed):
    """Both signs, exponent fields lo..hi (every one, the window's edges often), significands
    at random and at both ends of their range."""
    rng = np.random.default_rng(seed)
    e = rng.integers(lo, hi + 1, n)
    e[:hi - lo + 1] = np.arange(lo, hi + 1)
    e[-2000:] = np.tile([max(lo, 63), 64, 1983, min(hi, 1984)], 500)
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    m[::7] &= np.uint64(0xff)
    m[3::7] |= np.uint64((1 << 52) - 256)
    s = rng.integers(0, 2, n, dtype=np.uint64)
    return (s << np.uint64(63) | e.astype(np.uint64) << np.uint64(52) | m).view(np.float64)


def _reciprocals(a, n):
    nz = a.size // n
    D = np.zeros((nz, n, n))
    i = np.arange(n)
    D[:, i, i] = a.reshape(nz, n)
    zero = np.zeros((nz, n))
    rc, x = _call(D, zero, zero, np.ones((nz, n)))
    assert rc == 0
    return x.ravel()


@pytest.mark.parametrize('n,size,lo,hi', [(1, 40000, 1, 2046), (1, 8, 1000, 1003), (32, 32000, 4, 2040)])
def test_error_and_edges(n, size, lo, hi):
    a = _values(max(size, 4000), lo, hi, n + size)[:size]
    x = _reciprocals(a, n)
    field = (a.view(np.uint64) >> np.uint64(52) & np.uint64(0x7ff)).astype(int)
    inside = (field >= 64) & (field <= 1983)
    np.testing.assert_array_equal(x[~inside], 1.0 / a[~inside])
    ulp = np.spacing(np.abs(1.0 / a))
    worst = max(float(abs(Fraction(v) - 1 / Fraction(w)) / Fraction(u))
                for v, w, u in zip(x[inside].tolist(), a[inside].tolist(), ulp[inside].tolist()))
    print('n %d: %.4f ulp' % (n, worst))
    assert worst <= 0.57


def test_outside_the_normal_range():
    finite = np.array([np.inf, -np.inf, 2.0 ** -1023, -(2.0 ** -1024) * 1.5, 1.7e308, 2.0 ** 1023])
    overflow = np.array([5e-324, -1e-310])       # alone: times a coupling of zero they would be NaN
    with np.errstate(over='ignore'):
        for a in [finite, np.concatenate([finite, finite])] + [overflow[i:i + 1] for i in range(2)]:
            np.testing.assert_array_equal(_reciprocals(a, 1), 1.0 / a)
