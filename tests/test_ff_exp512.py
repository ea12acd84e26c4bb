"""The 512-entry float-float exponential of the MBIS "ff" kernels (exp_ff512 in
hp_ff.cuh), replayed in NumPy float32 arithmetic, against extended precision."""

import numpy as np
import pytest

f32 = np.float32
C1, C2, C3 = (f32(float.fromhex(c)) for c in ("0x1.62e43p-10", "-0x1.05c61p-38", "-0x1.950d88p-63"))
TABLE = [(f32(v), f32(v - np.longdouble(f32(v)))) for v in np.exp2(np.arange(512, dtype=np.longdouble) / 512)]


def fma(a, b, c):
    return f32(np.longdouble(np.float64(a) * np.float64(b)) + np.longdouble(c))


def two_sum(a, b):
    s = f32(a + b)
    bb = f32(s - a)
    return s, f32(f32(a - f32(s - bb)) + f32(b - bb))


def fast_two_sum(a, b):
    s = f32(a + b)
    return s, f32(b - f32(s - a))


def two_prod(a, b):
    p = f32(a * b)
    return p, fma(a, b, -p)


def exp_ff512(xh, xl):
    nf = f32(np.rint(f32(xh * f32(738.6598609))))
    n = int(nf)
    ph, pl = two_prod(nf, C1)
    ah, al = two_sum(xl, -pl)
    fh, fl = two_sum(f32(xh - ph), ah)
    fh, fl = fast_two_sum(fh, f32(fl + fma(-nf, C2, fma(-nf, C3, al))))
    sh, sl = two_prod(fh, fh)
    hh, hl = fast_two_sum(fh, f32(f32(0.5) * sh))
    low = fma(fh, fl, fl)
    low = fma(f32(0.5), sl, low)
    low = fma(f32(fh * sh), fma(fh, f32(1 / 24), f32(1 / 6)), low)
    low = f32(low + hl)
    tx, ty = TABLE[n & 511]
    qh, ql = two_prod(tx, hh)
    s0, s1 = fast_two_sum(tx, qh)
    r = f32(fma(tx, low, fma(ty, hh, ql)) + ty)
    vh, vl = fast_two_sum(s0, f32(s1 + r))
    return (np.longdouble(vh) + np.longdouble(vl)) * np.longdouble(2) ** (n >> 9)


@pytest.mark.parametrize("lo,hi", [(0.0, 1e-6), (1e-6, 1e-2), (1e-2, 1.0), (1.0, 20.0), (20.0, 60.0)])
def test_relative_error(lo, hi):
    rng = np.random.default_rng(3)
    for x in -rng.uniform(lo, hi, 800):
        xh = f32(x)
        xl = f32(x - np.float64(xh))
        want = np.exp(np.longdouble(xh) + np.longdouble(xl))
        # the rounding of n C2 (2^-24 of 4e-12 n) beside a few 2^-48 of the pairs
        assert abs(exp_ff512(xh, xl) / want - 1) < 1e-14 + 2e-16 * abs(x)
