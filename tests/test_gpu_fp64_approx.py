"""The FP64 reciprocal and inverse square root of the kernels against correctly rounded
values (extended precision), over random mantissas at every exponent where the path
changes, and over all exponents.

Bounds from the functions' derivation: 1 / d within 0.57 units in the last place, d^-1/2
within 1.1 (the library's own rsqrt: one unit); what takes the library's function gives
what that gives.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(exponents, n, seed):
    r = np.random.default_rng(seed)
    m = np.concatenate([r.integers(0, 1 << 52, n, dtype=np.uint64),
                        np.array([0, 1, (1 << 52) - 1, 1 << 51], dtype=np.uint64)])
    e = np.asarray(exponents, dtype=np.uint64)
    return ((e[:, None] << np.uint64(52)) | m[None]).reshape(-1).view(np.float64)


def _ulps(got, exact):
    """|got - exact| in units in the last place of the exact value."""
    rounded = exact.astype(np.float64)
    return (np.abs(got.astype(np.longdouble) - exact) / np.spacing(np.abs(rounded))).max()


@pytest.mark.parametrize("exponents,n", [((1, 2, 3, 4, 1022, 1023, 1024), 4000),
                                         ((2042, 2043, 2044), 4000), (range(1, 2045), 40)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_recip(ctx, exponents, n, sign):
    d = sign * _values(exponents, n, 1)
    assert _ulps(ctx.selftest_fp64("recip", d), 1 / d.astype(np.longdouble)) <= 0.57


@pytest.mark.parametrize("exponents,n", [((1, 2, 3, 4, 1022, 1023, 1024), 4000),
                                         ((2042, 2043, 2044, 2045, 2046), 4000),
                                         (range(1, 2047), 40)])
def test_rsqrt(ctx, exponents, n):
    d = _values(exponents, n, 2)
    assert _ulps(ctx.selftest_fp64("rsqrt", d), 1 / np.sqrt(d.astype(np.longdouble))) <= 1.1


def test_ends_of_the_range(ctx):
    """Results beyond exponent 2044 of the argument are subnormal: within half of the
    smallest; zeros, infinities, NaN and negative arguments as IEEE has them."""
    d = _values((2045, 2046), 400, 3)
    exact = 1 / d.astype(np.longdouble)
    got = ctx.selftest_fp64("recip", d)
    assert (np.abs(got.astype(np.longdouble) - exact) <= np.longdouble(2) ** -1075).all()
    tiny = np.array([5e-324, 2.0 ** -1074 * 3, 2.0 ** -1023, -2.0 ** -1060])
    with np.errstate(all="ignore"):
        for f, ref in (("recip", lambda x: 1 / x), ("rsqrt", lambda x: 1 / np.sqrt(x))):
            x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -2.0, -1e-300, -1e300])
            assert np.array_equal(ctx.selftest_fp64(f, x)[:5], ref(x)[:5], equal_nan=True)
            g = ctx.selftest_fp64(f, tiny)
            e = ref(tiny.astype(np.longdouble)).astype(np.float64)
            live = np.isfinite(e)
            assert np.array_equal(np.isfinite(g), live)
            assert (np.abs(g - e)[live] <= 1.1 * np.spacing(np.abs(e[live]))).all()
    assert np.isnan(ctx.selftest_fp64("rsqrt", np.array([-2.0, -1e-300, -1e300, -np.inf]))).all()
