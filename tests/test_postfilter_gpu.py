"""GPU: the DC blocker's block scan against the recursion as written, in double."""
import numpy as np
import pytest

from parallelfdtd_gb300 import postfilter as pf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 511, 512, 513, 8191, 8192, 8193, 17000])
@pytest.mark.parametrize("a", [0.995, 1.0, -0.7, 0.0, 1.0005])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_dc_block_equals_recursion(gpu, n, a, dtype):
    """y[t] = x[t] - x[t-1] + a y[t-1] at sizes around a thread's samples, a
    warp's and a tile's; |a| > 1 takes the serial kernel.  Each of the n sums
    of the chain rounds to at most eps of the largest partial sum, and the scan
    adds as many again, with the powers of a rounded on top: 4 n eps of the
    largest value; float results round once more."""
    x = np.random.default_rng(n).standard_normal((3, n)).astype(dtype)
    want = np.zeros((3, n))
    xp = yp = np.zeros(3)
    for t in range(n):
        yp = x[:, t].astype(np.float64) - xp + a * yp
        xp = x[:, t].astype(np.float64)
        want[:, t] = yp
    got = pf.fir(x, np.array([1.0]), dc_coef=a)
    assert got.dtype == dtype
    tol = 4 * n * np.finfo(np.float64).eps * np.abs(want).max()
    if dtype == np.float32:
        tol = tol + np.finfo(np.float32).eps * np.abs(want)
    assert np.all(np.abs(got.astype(np.float64) - want) <= tol)


@pytest.mark.parametrize("a", [0.995, 0.2, 0.0, -0.2, -0.7])
@pytest.mark.parametrize("at", [5, 16, 511, 9000])
@pytest.mark.parametrize("what", ["inf", "-inf", "nan", "overflow"])
def test_dc_block_not_finite(gpu, a, at, what):
    """A sample that is not finite, or a difference that overflows, leaves the
    recursion at the same infinities and NaNs for the rest of the trace, however
    far its powers of a have underflowed; before it the values are finite."""
    n = 20000
    x = np.random.default_rng(at).standard_normal(n)
    if what == "overflow":
        x[:at], x[at:] = -1.7e308, 1.7e308
    else:
        x[at] = float(what)
    want, xp, yp = np.zeros(n), 0.0, 0.0
    with np.errstate(all="ignore"):
        for t in range(n):
            yp = x[t] - xp + np.float64(a) * yp
            xp = x[t]
            want[t] = yp
    got = pf.fir(x[None], np.array([1.0]), dc_coef=a)[0]
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want))
    assert np.array_equal(np.isneginf(got), np.isneginf(want))


@pytest.mark.parametrize("channels,n", [(3, 699), (3, 700), (3, 701), (3, 719), (3, 720), (3, 721), (3, 1023),
                                        (3, 1024), (3, 1025), (3, 8207), (3, 8208), (3, 8209), (3, 8704),
                                        (152, 1000), (153, 1000), (200, 9000), (2000, 300), (5000, 40)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_dc_block_by_size(gpu, channels, n, dtype):
    """Few long traces take the block scan, many or short ones a thread each: at
    sizes on both sides of that line (700 samples of a few channels), of a
    thread's samples and of a warp's.  Tolerance as above."""
    a = 0.995
    x = np.random.default_rng(n).standard_normal((channels, n)).astype(dtype)
    want = np.zeros((channels, n))
    xp = yp = np.zeros(channels)
    for t in range(n):
        yp = x[:, t].astype(np.float64) - xp + a * yp
        xp = x[:, t].astype(np.float64)
        want[:, t] = yp
    got = pf.fir(x, np.array([1.0]), dc_coef=a)
    tol = 4 * n * np.finfo(np.float64).eps * np.abs(want).max()
    if dtype == np.float32:
        tol = tol + np.finfo(np.float32).eps * np.abs(want)
    assert np.all(np.abs(got.astype(np.float64) - want) <= tol)
