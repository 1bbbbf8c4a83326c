"""The envelope kernel at the edges of its tiles and passes (GPU), for even
lengths (whose even-offset taps are exactly zero and are skipped) and odd
ones: against the circular convolution evaluated with NumPy in float64, a
bound of N rounding errors on the sum of |x| |g|; and samples that are not
finite, which make every output of a skipped product NaN as the product with
the zero tap would be."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _taps(n):
    m = np.arange(1, n)
    g = np.zeros(n)
    if n % 2 == 0:
        g[1:] = np.where(m % 2, 2.0 / n / np.tan(np.pi * m / n), 0.0)
    else:
        g[1:] = (1 / np.tan(np.pi * m / n) - (-1.0) ** m / np.sin(np.pi * m / n)) / n
    return g


@pytest.mark.parametrize("lens", [[1, 2, 3, 4], [510, 511, 512, 513, 514], [1023, 1024, 1025, 1026, 1024], [2050, 1537]])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_tiles_and_passes(lens, dtype):
    from pefdtd import traces
    rng = np.random.default_rng(1)
    xs = [rng.normal(size=n).astype(dtype) for n in lens]
    for x, e in zip(xs, traces.envelope(xs)):
        n, g = len(x), _taps(len(x))
        x = x.astype(float)
        h = np.array([np.dot(x, g[(k - np.arange(n)) % n]) for k in range(n)])
        want = np.hypot(x, h)
        # n products and sums, and a tap's own evaluation, each within a few ulp
        bound = 4 * (n + 8) * np.finfo(float).eps * np.abs(x).sum() * max(np.abs(g).max(), 1.0)
        assert np.abs(e - want).max() <= bound


@pytest.mark.parametrize("n", [6, 7, 600, 601])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_samples_that_are_not_finite(n, bad):
    from pefdtd import traces
    x = np.ones(n)
    x[3] = bad
    e = traces.envelope(x)
    d = (np.arange(n) - 3) % n
    if np.isnan(bad):
        assert np.isnan(e).all()
    else:   # the sample itself: |inf|; zero taps (cot(pi / 2) is one): inf * 0; the others: inf
        zero = (d % 2 == 0) | (2 * d == n) if n % 2 == 0 else (d == 0)
        want = np.where(d == 0, np.inf, np.where(zero, np.nan, np.inf))
        assert np.array_equal(e, want, equal_nan=True)
