"""The device's own elementary functions, evaluated on the GPU against extended precision."""

import numpy as np
import pytest

import device_checks

pytestmark = pytest.mark.gpu


def _random(rng, lo, hi, n=200000):
    return -rng.uniform(lo, hi, n) if lo == 0.0 else -np.exp(rng.uniform(np.log(lo), np.log(hi), n))


@pytest.mark.parametrize("lo,hi", [(0.0, 1e-6), (1e-6, 1e-2), (1e-2, 1.0), (1.0, 20.0), (20.0, 40.0), (40.0, 60.0),
                                   (60.0, 86.99)])
def test_exp_ff512(lo, hi):
    x = _random(np.random.default_rng(3), lo, hi)
    xh = x.astype(np.float32).astype(np.float64)
    xl = (x - xh).astype(np.float32).astype(np.float64)
    with np.errstate(under="ignore"):
        want = np.exp(xh.astype(np.longdouble) + xl)
    err = {}
    for what in ("exp_ff512", "exp_ff"):
        v, l = device_checks.evaluate(what, xh, xl)
        err[what] = (v.astype(np.longdouble) + l - want).astype(np.float64)
    # three roundings of the low part, 2^-25 of at most 2^-23 each: 1.1e-14; the low part ends at 2^-149
    assert np.all(np.abs(err["exp_ff512"]) <= 1.1e-14 * want + 2.0**-149)
    rms = {k: np.sqrt(np.mean(np.square(e / want.astype(np.float64)))) for k, e in err.items()}
    assert rms["exp_ff512"] <= rms["exp_ff"]


def test_exp_ff512_edges():
    x = np.array([0.0, -0.0, -87.0, np.nextafter(np.float32(-87), np.float32(-88)), -100.0, -np.inf, 1.0, 80.0])
    v, l = device_checks.evaluate("exp_ff512", x)
    want = np.exp(x.astype(np.longdouble))
    want[3:6] = 0.0  # below the FP32 normal range
    assert np.all(np.abs(v.astype(np.longdouble) + l - want) <= 1.1e-14 * want + 2.0**-149)


def _ulps(got, want):
    """Errors in units of the last place of the rounded result (2^-1074 at least)."""
    return np.abs((got.astype(np.longdouble) - want) / np.spacing(np.abs(want.astype(np.float64))))


def _scaled(rng, n, lo, hi):
    return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n, endpoint=True))


@pytest.mark.parametrize("lo,hi,ulps", [(1e-300, 1e-3, 1.02), (1e-3, 1.0, 1.02), (1.0, 100.0, 1.02), (100.0, 707.99, 1.02),
                                        (708.0, 745.0, 2.0)])  # the last range is CUDA's exp
@pytest.mark.parametrize("sign", [-1.0, 1.0])
def test_exp64(sign, lo, hi, ulps):
    x = -sign * _random(np.random.default_rng(5), lo, hi)
    x = x[x < 709.7]
    x = np.concatenate([x, np.nextafter(sign * np.array([708.0, 708.0]), [-1e3, 1e3])]) if hi > 700.0 else x
    got = device_checks.evaluate("exp64", x)[0]
    assert np.max(_ulps(got, np.exp(x.astype(np.longdouble)))) < (2.0 if hi > 700.0 else ulps)


def test_exp64_edges():
    inf, nan = np.inf, np.nan
    x = np.array([0.0, -0.0, 5e-324, -745.0, -745.2, -746.0, -1e4, -1e300, -inf, 709.0, 710.0, inf, nan, -nan])
    with np.errstate(over="ignore", under="ignore"):
        want = np.exp(x)
    got = device_checks.evaluate("exp64", x)[0]
    plain = np.isin(x, [0.0, 5e-324, -746.0, -1e4, -1e300, -inf, 710.0, inf]) | np.isnan(x)
    np.testing.assert_array_equal(got[plain], want[plain])
    np.testing.assert_array_less(_ulps(got[~plain], np.exp(x[~plain].astype(np.longdouble))).astype(float), 2.0)


def test_div64():
    rng = np.random.default_rng(6)
    n = 1 << 20
    for lo, hi in ((-20, 20), (-950, -900), (900, 960)):
        a, d = _scaled(rng, n, -40, 40), _scaled(rng, n, lo, hi)
        got = device_checks.evaluate("div64", a, d)[0]
        assert np.max(_ulps(got, a.astype(np.longdouble) / d)) < 1.52
    # on both sides of the guard 2^-959 <= d < 2^961, and what is divided plainly
    d = np.array([2.0**-959, np.nextafter(2.0**-959, 0), 2.0**961, np.nextafter(2.0**961, 0), 2.0**960, 2.0**-960, 1.0])
    for a in (0.0, 1.0, 3.0, -7.0, 1e-30):
        assert np.max(_ulps(device_checks.evaluate("div64", np.full(7, a), d)[0], a / d.astype(np.longdouble))) < 1.52
    d = np.array([0.0, -0.0, -1.5, 5e-324, np.inf, -np.inf, np.nan, 2.0])
    for a in (0.0, 1.0, -2.0, np.inf, np.nan):
        with np.errstate(all="ignore"):
            np.testing.assert_array_equal(device_checks.evaluate("div64", np.full(8, a), d)[0], a / d)


def test_rsqrt64():
    rng = np.random.default_rng(7)
    n = 1 << 20
    for lo, hi in ((-20, 20), (-955, -900), (900, 960)):
        d = _scaled(rng, n, lo, hi)
        assert np.max(_ulps(device_checks.evaluate("rsqrt64", d)[0], 1 / np.sqrt(d.astype(np.longdouble)))) < 1.03
    d = np.array([2.0**-959, np.nextafter(2.0**-959, 0), 2.0**961, np.nextafter(2.0**961, 0), 1e-300, 5e-324, 1e308])
    # sqrt and a division: two roundings, half an ulp each, up to one of the result
    assert np.max(_ulps(device_checks.evaluate("rsqrt64", d)[0], 1 / np.sqrt(d.astype(np.longdouble)))) < 1.52
    with np.errstate(all="ignore"):
        d = np.array([0.0, -1.0, np.inf, np.nan])
        np.testing.assert_array_equal(device_checks.evaluate("rsqrt64", d)[0], 1 / np.sqrt(d))


SPECIAL = np.array([0.0, -0.0, 5e-324, -5e-324, 1e-300, -1e-300, 1e-15, np.nextafter(1e-15, 0), np.nextafter(1e-15, 1), 0.5,
                    np.nextafter(1.0, 0), 1.0, np.nextafter(1.0, 2), 2.0, -1.0, -2.0, 1e300, -1e300, np.inf, -np.inf,
                    np.nan, -np.nan])


def test_clip01():
    x = np.concatenate([SPECIAL, np.random.default_rng(8).uniform(-1.0, 2.0, 5000)])
    want = np.where(np.isnan(x), 0.0, np.clip(x, 0.0, 1.0))  # fmin(fmax(x, 0), 1)
    np.testing.assert_array_equal(device_checks.evaluate("clip01", x)[0], want)


def test_below():
    x, c = (v.ravel() for v in np.meshgrid(SPECIAL, SPECIAL))
    np.testing.assert_array_equal(device_checks.evaluate("below", x, c)[0], (x < c).astype(float))
