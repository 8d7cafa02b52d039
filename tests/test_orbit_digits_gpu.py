"""The reference orbit against exact integers at every shape of its producer:
one to six warps, odd and even digit counts, the smallest and the largest, each
formula, and short orbits (that escape, or end at the last entry)."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal, native

pytestmark = pytest.mark.gpu


def exact_orbit(x, y, F, n, fractal):
    """Z_1 .. Z_n of z' = f(z) + c in F-bit fixed point, guard bits kept."""
    zs, X, Y = [(0, 0)], x, y
    for _ in range(n):
        zs.append((X, Y))
        if X * X + Y * Y > 4 << (2 * F):
            break
        re, im = (X * X - Y * Y) >> F, (2 * X * Y) >> F
        if fractal == 1:
            im = abs(im)
        if fractal == 2:
            re = abs(re)
        X, Y = re + x, im + y
    return zs


@pytest.mark.parametrize("limbs", [5, 7, 9, 12, 13, 14, 21, 26, 27, 29, 40, 41, 53, 54, 65, 68, 80])
@pytest.mark.parametrize("fractal", [0, 1, 2])
def test_orbit_digits(renderer, limbs, fractal):
    F, n = 28 * (limbs - 1), 60
    lib = native.load()
    # c = i (and near it) stays bounded; -0.6 + 0.2 i too; 0.5 + 0.5 i escapes
    for cx, cy in ((Fraction(0), Fraction(1)), (Fraction(-3, 5), Fraction(1, 5)),
                   (Fraction(1, 2), Fraction(1, 2))):
        vals = [MpVal.from_fraction(v, F) for v in (cx, cy)]
        s = [v.struct() for v in vals]
        x, y = (int(v.to_fraction() * 2 ** F // 1) for v in vals)
        for last in (1, 2, n):
            re, im = np.zeros(last + 1), np.zeros(last + 1)
            ln = C.c_int64()
            assert lib.mdzgpu_reference_orbit_formula(
                renderer.ctx, fractal, C.byref(s[0][0]), C.byref(s[1][0]), F, limbs, last,
                re.ctypes.data, im.ctypes.data, None, None, C.byref(ln)) == 0
            want = exact_orbit(x, y, F, last, fractal)
            assert ln.value == len(want)
            # a step drops columns below the fourth guard digit: under 2^(10 - F)
            # a step, growing by at most 4 a step; the rounding to double is 2^-53
            for k, (X, Y) in enumerate(want):
                err = 2.0 ** (10 - F + 2 * k) + 2.0 ** -50
                assert abs(re[k] - X / 2 ** F) <= err and abs(im[k] - Y / 2 ** F) <= err, (k, last)
