"""The warp-cooperative multi-limb kernel, bit for bit, at every word count:
counts on a chaotic view against the same truncated products in Python."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal, native

pytestmark = pytest.mark.gpu

WORDS = [48, 64, 80, 96, 128, 160, 192, 256]


def truncated(a, b, NL):
    """Sum of the partial products a_i b_j of 64-bit limbs with i + j >= NL-2."""
    s = 0
    for i in range(NL):
        cut = max(0, NL - 2 - i)
        s += (((a >> (64 * i)) & 0xffffffffffffffff) * (b >> (64 * cut))) << (64 * (i + cut))
    return s


def count(x, y, cx, cy, NL, depth, fractal):
    F = 64 * NL - 8
    re2, im2 = (truncated(abs(v), abs(v), NL) >> F for v in (x, y))
    for wz in range(1, depth + 1):
        t = (2 * truncated(abs(x), abs(y), NL)) >> F
        d = re2 - im2
        if fractal != 1 and (x < 0) != (y < 0):
            t = -t
        if fractal == 2 or (fractal == 3 and wz & 1):
            d = abs(d)
        x, y = cx + d, cy + t
        if any((v >> (64 * NL - 64)) >= 0x0800000000000000
               or (v >> (64 * NL - 64)) < -0x0800000000000000 for v in (x, y)):
            return wz
        re2, im2 = (truncated(abs(v), abs(v), NL) >> F for v in (x, y))
        if re2 + im2 > 4 << F:
            return wz
    return 0


@pytest.mark.parametrize("words", WORDS)
@pytest.mark.parametrize("W,H", [(5, 3), (1, 2)])
def test_mpw_counts_exact(renderer, words, W, H):
    k = WORDS.index(words)
    fractal, julia = (k + H) % 4, None
    if k % 3 == 2:
        julia = (MpVal.from_fraction(Fraction(-4, 5), 64), MpVal.from_fraction(Fraction(39, 250), 64))
    prec, depth = 32 * words - 8, 100
    span = MpVal.from_fraction(Fraction(1, 2 ** (prec - 12)), prec)
    # near c = 1/4 i: stays bounded a while under every formula
    xmin = MpVal.from_fraction(Fraction(-7436447860, 10 ** 10), prec)
    ymax = MpVal.from_fraction(Fraction(1318252536, 10 ** 10), prec)
    got, st = renderer.render_mp(W, H, depth, xmin, ymax, span, prec, words=words, fractal=fractal,
                                 family=1 if julia else 0, julia=julia)
    assert st["words"] == words
    lib = native.load()
    tab = np.zeros((W + H, words), np.uint32)
    s = [v.struct() for v in (xmin, ymax, span)]
    assert lib.mdzgpu_mp_coordinates(*[C.byref(v) for v, _ in s], W, 0, H, prec, words,
                                     tab.ctypes.data, tab[W:].ctypes.data) == 0
    num = [int.from_bytes(r.tobytes(), "little", signed=True) for r in tab]
    F = 32 * words - 8
    jc = [int(v.to_fraction() * 2 ** F // 1) for v in julia] if julia else None
    want = np.array([[count(num[ix], num[W + r], *(jc or (num[ix], num[W + r])), words // 2, depth,
                            fractal) for ix in range(W)] for r in range(H)], np.int32)
    assert np.array_equal(got, want)
