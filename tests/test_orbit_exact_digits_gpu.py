"""Every digit of the reference orbits against a restatement in whole numbers:
the kept columns of Z_k^2, the two carry passes, the folds, C.

All shapes of the producer (one to six warps of 14 columns), the streamed orbit
and the one made before the frame, the Julia family's two orbits (one from a
given Z_0) and the hybrid's two (folds at odd and at even steps)."""
import ctypes as C
import random
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal

pytestmark = pytest.mark.gpu

DEPTH = 50


def split(v):
    d = ((v + (1 << 27)) & ((1 << 28) - 1)) - (1 << 27)
    return d, (v - d) >> 28


def carry_twice(cols):
    for _ in range(2):
        parts = [split(v) for v in cols]
        cols = [d + (parts[i - 1][1] if i else 0) for i, (d, _) in enumerate(parts)]
    return cols


def sign(digits):
    top = [d for d in digits if d]
    return 0 if not top else 1 if top[-1] > 0 else -1


def step(x, y, cx, cy, fractal, folds):
    """Digits of Z' from those of Z; columns L-4 .. 2L-2 are kept."""
    L = len(x)
    re, im = [], []
    for c in range(L - 4, 2 * L - 1):
        pairs = [(i, c - i) for i in range(max(0, c - L + 1), min(c, L - 1) + 1)]
        re.append(sum(x[i] * x[j] - y[i] * y[j] for i, j in pairs))
        im.append(2 * sum(x[i] * y[j] for i, j in pairs))
    add = lambda cols, c: [v + (c[k - 3] if k >= 3 else 0) for k, v in enumerate(cols)]
    if fractal == 1:
        s = sign(x) * sign(y)
        im = [s * v for v in im]
    if folds:
        re = carry_twice(re)
        if sign(re) < 0:
            re = [-v for v in re]
    return carry_twice(add(re, cx))[3:], carry_twice(add(im, cy))[3:]


def orbits(renderer, L):
    found = []
    for which in (0, 1):
        limbs, n = C.c_int32(), C.c_int64()
        d = np.zeros((DEPTH + 2, 2, L), np.int32)
        if renderer.lib.mdzgpu_last_orbit_digits(renderer.ctx, which, d.ctypes.data, len(d),
                                                 C.byref(limbs), C.byref(n)):
            break
        assert limbs.value == L
        found.append(d[:n.value].tolist())
    return found


def check(orbit, cx, cy, fractal, parity=None):
    assert len(orbit) > 10
    for k in range(len(orbit) - 1):
        x, y = orbit[k]
        folds = fractal == 2 or (parity is not None and k % 2 == parity)
        want = step(x, y, cx, cy, fractal, folds)
        assert orbit[k + 1] == [want[0], want[1]], k


# one to six warps: up to 12, 26, 40, 54, 68, 80 digits
LIMBS = [5, 7, 9, 12, 13, 14, 21, 26, 27, 29, 40, 41, 53, 54, 55, 65, 68, 69, 80]


@pytest.mark.parametrize("limbs", LIMBS)
@pytest.mark.parametrize("kind", ["mandelbrot", "ship", "celtic", "hybrid", "julia",
                                  "julia-ship", "julia-celtic"])
def test_every_digit(renderer, monkeypatch, kind, limbs):
    F = 28 * (limbs - 1)
    rng = random.Random(limbs)
    # the low bits at random: every digit is in use from the first step on
    near = lambda v: Fraction((round(v * 2 ** 24) << (F - 24)) + rng.getrandbits(F - 24), 2 ** F)
    val = lambda v: MpVal.from_fraction(v, F)
    fractal = 3 if kind == "hybrid" else ["mandelbrot", "ship", "celtic"].index(
        kind.split("-")[-1].replace("julia", "mandelbrot"))
    centre = val(near(-0.3)), val(near(0.2))
    julia = (val(near(-0.4)), val(near(0.15))) if kind.startswith("julia") else None
    for schedule in ("steps", "frame"):
        monkeypatch.setenv("MDZGPU_PERTURB", schedule)
        renderer.render_perturb(8, 4, DEPTH, *centre, val(Fraction(1, 2 ** 12)), F, limbs=limbs,
                                fractal=fractal, julia=julia)
        got = orbits(renderer, limbs)
        assert len(got) == (2 if kind == "hybrid" or julia else 1)
        if julia:
            cx, cy = got[1][1]    # Q_0 = 0, Q_1 = C
            assert got[1][0] == [[0] * limbs] * 2
            check(got[0], cx, cy, fractal)
            check(got[1], cx, cy, fractal)
            start, want = got[0][0], centre
        else:
            cx, cy = start = got[0][1]
            want = centre
            for parity, orbit in zip((1, 0), got):
                assert orbit[0] == [[0] * limbs] * 2 and orbit[1] == [cx, cy]
                check(orbit[1:], cx, cy, fractal,
                      None if kind != "hybrid" else 1 - parity)
        for digits, v in zip(start, want):
            assert sum(d << (28 * j) for j, d in enumerate(digits)) == v.to_fraction() * 2 ** F
