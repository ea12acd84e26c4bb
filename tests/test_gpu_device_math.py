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
