"""The day step's fixed-point exp, pow and reciprocal at the edges of their
ranges: interval boundaries of the tables, both sides of a power of two and of 1,
the changes of scale of the logarithm (2^-16, 2^-128), tiny and large exponents,
and arguments that are not finite.

Bounds in ulp of the result, from the error terms: half an ulp of the final
rounding plus, for exp, four units of |x| log2(e) to 62 bits (below 2^-57 for
|x| < 32, 2^-4 ulp); for pow, eight units of y log2(x), whose format keeps
64 - (integer bits of log2 x) - (those of y) bits after the point."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
needs_quad = pytest.mark.skipif(np.finfo(LD).nmant < 63, reason="no wider type to compare with")


def _ulp(got, ref):
    return np.abs(LD(got) - ref) / np.spacing(np.abs(ref).astype(np.float64)).astype(LD)


def _around(x):
    x = np.asarray(x, np.float64)
    return np.concatenate([np.nextafter(x, -np.inf), x, np.nextafter(x, np.inf)])


@needs_quad
def test_exp_at_interval_edges():
    from watergap2_gb300.gpu import math_eval
    k = np.arange(-46 * 256, 46 * 256)
    x = np.concatenate([_around(k * (np.log(2.0) / 256)), np.logspace(-20, 0, 500), -np.logspace(-20, 0, 500)])
    x = x[np.abs(x) < 32]
    assert _ulp(math_eval("exp", x), np.exp(LD(x))).max() < 0.5 + 2.0 ** -4
    big = np.concatenate([np.linspace(32, 709, 3000), -np.linspace(32, 708, 3000)])
    assert _ulp(math_eval("exp", big), np.exp(LD(big))).max() < 0.75


@needs_quad
@pytest.mark.parametrize("y", [0.001, 0.1, 0.341, 0.66666666, 2.0 / 3.0, 1.0, 2.5, 7.9, 8.0, 300.0])
def test_pow_at_interval_edges(y):
    from watergap2_gb300.gpu import math_eval
    j = 1.0 + np.arange(256) / 256.0
    x = np.concatenate([_around(np.ldexp(j, e)) for e in (-200, -129, -128, -17, -16, -1, 0, 1, 15, 16, 100)])
    x = np.concatenate([x, 1.0 - np.logspace(-16, -1, 200), 1.0 + np.logspace(-15, -1, 200)])
    x = x[np.abs(y * np.log2(x)) < 1000]
    ref = LD(x) ** LD(y)
    whole = np.where(np.abs(np.log2(x)) < 17, 5, np.where(np.abs(np.log2(x)) < 129, 8, 12))
    whole = whole + max(int(np.floor(np.log2(y))) + 1, -4)
    bound = 0.5 + 2.0 ** -4 + 8 * np.ldexp(0.7, 53 + whole - 64)
    assert np.all(_ulp(math_eval("pow", x, y), ref) < bound)


@needs_quad
def test_reciprocal_at_powers_of_two():
    from watergap2_gb300.gpu import math_eval
    x = np.concatenate([_around(np.ldexp(1.0, np.arange(-1000, 1000))), _around(1.0 + np.arange(1, 512) / 512.0)])
    x = np.concatenate([x, -x])
    assert _ulp(math_eval("rcp", x), 1 / LD(x)).max() < 0.51


def test_arguments_outside_the_ranges():
    from watergap2_gb300.gpu import math_eval
    inf, nan = np.inf, np.nan
    x = np.array([0.0, -0.0, 5e-324, -5e-324, inf, -inf, nan, 710.0, -745.2, -746.0, 1e300, -1e300])
    with np.errstate(all="ignore"):
        assert np.array_equal(math_eval("exp", x), np.exp(x), equal_nan=True)
        deep = np.linspace(-745, -708.5, 500)          # subnormal results
        assert np.all(np.abs(math_eval("exp", deep) - np.exp(deep)) <= 5e-324)
    px = np.array([0.0, -0.0, -2.0, 1.0, 2.0, 0.5, 2.0, 0.5, 2.0, inf, 3.0])
    py = np.array([0.5, 0.5, 0.5, 9.0, 1e300, 1e300, -1e300, -1e300, 1024.0, 0.5, 0.0])
    want = np.array([0.0, 0.0, 0.0, 1.0, inf, 0.0, 0.0, inf, inf, inf, 1.0])
    assert np.array_equal(math_eval("pow", px, py), want)
    assert np.isnan(math_eval("pow", np.array([2.0, nan]), np.array([nan, 2.0]))).all()
    assert np.isnan(math_eval("rcp", np.array([0.0, inf, nan]))).all()
