"""The multi-limb frame kernel, bit for bit: counts on a chaotic view (where
a unit in the last place changes them) against the same truncated products in
Python integers, at every word count, on frames whose tiles are ragged."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal, native

pytestmark = pytest.mark.gpu

WORDS = [4, 6, 8, 10, 12, 16, 20, 24, 28, 34, 36]


def truncated(a, b, N):
    """Sum of the partial products a_i b_j of 32-bit words with i + j >= N-2."""
    s = 0
    for i in range(N):
        cut = max(0, N - 2 - i)
        s += (((a >> (32 * i)) & 0xffffffff) * (b >> (32 * cut))) << (32 * (i + cut))
    return s


def count(x, y, cx, cy, N, depth, fractal):
    """Escape iteration (0: none) of the kernel's loop: magnitudes multiplied,
    truncated below column N-2, shifted down F = 32 N - 8 bits."""
    F = 32 * N - 8
    re2, im2 = (truncated(abs(v), abs(v), N) >> F for v in (x, y))
    for wz in range(1, depth + 1):
        t = (2 * truncated(abs(x), abs(y), N)) >> F
        d = re2 - im2
        if fractal != 1 and (x < 0) != (y < 0):
            t = -t
        if fractal == 2 or (fractal == 3 and wz & 1):
            d = abs(d)
        x, y = cx + d, cy + t
        if any(v >= 8 << F or v < -(8 << F) for v in (x, y)):
            return wz
        re2, im2 = (truncated(abs(v), abs(v), N) >> F for v in (x, y))
        if re2 + im2 > 4 << F:
            return wz
    return 0


@pytest.mark.parametrize("words", WORDS)
@pytest.mark.parametrize("W,H", [(9, 5), (33, 1), (1, 6)])
def test_mp_counts_exact(renderer, words, W, H):
    k = WORDS.index(words)
    fractal, julia = k % 4, None
    if k % 3 == 2 or H == 1:
        julia = (MpVal.from_fraction(Fraction(-4, 5), 64), MpVal.from_fraction(Fraction(39, 250), 64))
    prec, depth = 32 * words - 8, 90 if words > 20 else 200
    # a view a few last places wide across an orbit that stays bounded long
    span = MpVal.from_fraction(Fraction(1, 2 ** (prec - 12)), prec)
    cx, cy = Fraction(-7436447860, 10 ** 10), Fraction(1318252536, 10 ** 10)
    xmin, ymax = MpVal.from_fraction(cx, prec), MpVal.from_fraction(cy, prec)
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
    want = np.array([[count(num[ix], num[W + r], *(jc or (num[ix], num[W + r])), words, depth,
                            fractal) for ix in range(W)] for r in range(H)], np.int32)
    assert np.array_equal(got, want)
