"""The element kernels' reciprocal (csrc/dg_roe_ff.cuh, rcp_seeded) on the device, against its error bound and the
correctly rounded one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
dp = C.POINTER(C.c_double)


def _both(pkg, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    f = pkg.lib().dg_reciprocal_nodes
    f.restype, f.argtypes = C.c_int, [C.c_int, dp, dp, dp]
    a, b = np.empty_like(x), np.empty_like(x)
    assert f(x.size, *[v.ctypes.data_as(dp) for v in (x, a, b)]) == 0
    return a, b


@pytest.mark.parametrize("scale", [0, -100, -37, 99])
def test_reciprocal_within_its_bound(pkg, scale):
    """0.5 + 2^-12 units in the last place for any significand (the cut term and the roundings before the last
    are below 2^-65 of the value together), which a correctly rounded one exceeds 0.5 by nothing."""
    rng = np.random.default_rng(abs(scale))
    n = 400000
    m = np.concatenate([rng.uniform(1, 2, n), 1 + np.arange(2000) * 2.0 ** -52, 2 - np.arange(1, 2000) * 2.0 ** -52,
                        1 + rng.integers(0, 1 << 24, 2000) * 2.0 ** -24, 1 + (rng.integers(1, 1 << 24, 2000) * 2.0 ** 29 - 1) * 2.0 ** -52])
    x = np.ldexp(m * rng.choice([-1.0, 1.0], m.size), scale)
    a, b = _both(pkg, x)
    # the residual (a - 1/x) / ulp(a) = (a x - 1) / (x ulp(a)), a x - 1 exactly from 26-bit halves
    def halves(v):
        h = (v.view(np.int64) & ~np.int64((1 << 27) - 1)).view(np.float64)
        return h, v - h
    xh, xl = halves(x)
    for y, tol in ((a, 0.5 + 2.0 ** -12), (b, 0.5)):
        yh, yl = halves(y)
        r = (((yh * xh - 1.0) + yh * xl) + yl * xh) + yl * xl
        ulp = np.abs(r / (x * np.spacing(np.abs(y))))
        assert float(ulp.max()) <= tol + 2.0 ** -20
    assert np.mean(a != b) < 1e-3


def test_reciprocal_elsewhere_is_the_rounded_one(pkg):
    """Outside 2^-100 .. 2^100: zeros, subnormals, the ends of the range, infinities and NaN."""
    x = np.array([0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1022, 2.0 ** -1023, 2.0 ** -101, -1.5 * 2.0 ** -101, 2.0 ** 100, 2.0 ** 101,
                  -2.0 ** 512, 1.7976931348623157e308, np.inf, -np.inf, np.nan])
    a, b = _both(pkg, x)
    assert np.array_equal(a.view(np.int64)[:-1], b.view(np.int64)[:-1]) and np.isnan(a[-1])
    with np.errstate(all="ignore"):
        assert np.array_equal((1.0 / x).view(np.int64)[:-1], b.view(np.int64)[:-1])
