"""The inner products of BiCGStab on vectors whose products cancel, against the
exact sum: they are carried as pairs hi + lo, with which (v, rp) and (r, rp) keep
their digits far below the size of their terms."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS, CTAS = 256, 296


def _split(a):
    c = 134217729.0 * a
    hi = c - (c - a)
    return hi, a - hi


def _two_product(x, y):
    """x y = p + e exactly (Veltkamp's splitting, Dekker's product)."""
    p = x * y
    xh, xl = _split(x)
    yh, yl = _split(y)
    return p, xl * yl - (((p - xh * yh) - xl * yh) - xh * yl)


def _exact(x, y):
    p, e = _two_product(x, y)
    return math.fsum(np.concatenate([p, e]).tolist())


def _cancelling(n, seed):
    """Vectors whose product falls to about 1e-18 of its terms: random ones, then terms that take off what is there so far."""
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    last = min(n // 2, 40)
    for k, i in enumerate(range(n - last, n)):
        s = 2.0 ** (-60.0 * (k + 1) / last)
        x[i] *= s ** 0.5
        x[i] += math.copysign(0.1 * s ** 0.5, x[i])
        y[i] = (s * rng.uniform(0.5, 1) - _exact(x[:i], y[:i])) / x[i]
    order = rng.permutation(n)
    return x[order], y[order]


@pytest.mark.parametrize("n", [2, 33, 363, 1024, 1025, 6912, 150001, 310003])
def test_products_keep_their_digits_under_cancellation(n):
    """A pair's hi is exact but for lo, and lo adds up d + 1 errors of at most u times the sum of the magnitudes m,
    each addition rounding at u: at most 2 (d + 2)^2 u^2 m for sums of depth d, and u for each of the rounding of the
    pair and the quotient.  A plain sum, or a product whose error is added twice, is off by about u m."""
    v, w = _cancelling(n, n)
    (alpha, reason), (omega, _) = _run(v, w)
    exact = _exact(v, w)
    m = float(np.abs(v * w).sum())
    u = 2.0 ** -53
    grid = min(CTAS, max(1, -(-n // (4 * THREADS))))
    depth = -(-n // (grid * THREADS)) + 5 + THREADS // 32 + -(-grid // THREADS) + 5 + THREADS // 32
    bound = 2 * (depth + 2) ** 2 * u * u * m
    assert n < 300 or abs(exact) > 100 * bound                       # the case says something
    assert n < 300 or abs(exact) < 0.01 * u * m
    assert reason == 0
    assert abs(1.0 / alpha - exact) <= bound + 3 * u * abs(exact)
    ww = _exact(w, w)
    assert abs(omega * ww - exact) <= bound + 5 * u * abs(exact)


@pytest.mark.parametrize("n", [2, 5000])
def test_overflow_and_nan_end_as_in_a_plain_sum(n):
    """(w, w) = inf and (v, w) finite: omega = 0; infinite or undefined (v, w): KSP_DIVERGED_NANORINF; zero: breakdown."""
    v, w = np.zeros(n), np.zeros(n)
    v[[0, -1]], w[[0, -1]] = [1.0, 2.0], [1e200, 1e10]
    assert _run(v, w) == ((1.0 / (1e200 + 2e10), 0), (0.0, 0))
    assert _run(-v, w)[1] == (0.0, 0)
    v[0] = 1e200
    assert _run(v, w)[0] == (None, -9)
    for bad in (np.inf, np.nan):
        v[0], w[0] = bad, 1.0
        assert _run(v, w)[0] == (None, -9)
    v[[0, -1]], w[[0, -1]] = [0.0, 1.0], [1.0, 0.0]
    assert _run(v, w) == ((None, -5), (0.0, 0))


def _run(v, w):
    from cfdsfemmpi_b200._lib import bcgs_scalars
    return bcgs_scalars(v, w)
