"""Multi-limb frames large enough that lanes are refilled and that warps move
their pixels together at the end: each row's counts are those of the row as a
frame of its own (fewer than one tile a block, so neither happens there).  The
coordinates are dyadic, so both frames' are exact."""
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words,fractal,julia", [
    (4, 0, None), (10, 1, None), (16, 2, None), (16, 0, (-0.8, 0.15625)), (20, 3, None),
    (28, 1, None), (34, 0, None), (36, 2, None)])
def test_rows_of_a_large_frame(renderer, words, fractal, julia):
    W, H, depth = 512, 164, 700 if words < 20 else 250
    prec = 32 * words - 8
    q = lambda v: MpVal.from_fraction(Fraction(v), prec)
    kw = dict(words=words, fractal=fractal, family=1 if julia else 0,
              julia=tuple(q(v) for v in julia) if julia else None)
    top, x0, width = Fraction(5, 8), Fraction(-9, 4), Fraction(4)
    full = np.array(renderer.render_mp(W, H, depth, q(x0), q(top), q(width), prec, **kw)[0])
    assert len(np.unique(full)) > 20
    for line in (0, 1, 40, 80, 123, H - 1):
        row = renderer.render_mp(W, 1, depth, q(x0), q(top - width * line / W), q(width), prec,
                                 **kw)[0]
        assert np.array_equal(row[0], full[line]), line
