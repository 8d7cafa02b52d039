"""The smallest depths through MDZ's own entry points, which take any: a pixel
that escapes after n iterations has count n from depth n on and 0 below it, so
depths of 0 and less give a frame of zeros (the reference's loop is
wz = 1 .. depth).  Double, MPFR and GMP callbacks, a precision of the
warp-cooperative kernel, and the line functions."""
import ctypes as C

import numpy as np
import pytest

from mdz_gb300 import View
from mdz_gb300.abi import DropIn

pytestmark = pytest.mark.gpu

# multi_prec, rounding, precision, line function
PATHS = [(0, 0, 80, "fractal_calculate_line"), (1, 1, 80, "fractal_mpfr_calculate_line"),
         (1, 0, 128, "fractal_gmp_calculate_line"), (1, 1, 1300, "fractal_mpfr_calculate_line")]


def counts(path, depth, line=None):
    v = View("small", 37, 21, 1, "-0.5", "0.1", "4", precision=path[2], multi_prec=path[0],
             rounding=path[1])
    d = DropIn(v)
    try:
        d.img.depth = depth
        if line is None:
            d.render(timeout_s=60)
            return d.raw.copy()
        assert getattr(d.lib, path[3])(C.byref(d.img), line) == 1
        return d.raw[line].copy()
    finally:
        d.close()


@pytest.mark.parametrize("path", PATHS, ids=["double", "mpfr80", "gmp", "mpfr1300"])
def test_small_depths(path):
    full = counts(path, 40)
    assert len(np.unique(full)) > 8 and full.min() == 0
    for depth in (-2 ** 40, -1, 0, 1, 2, 3, 5):
        want = np.where(full <= depth, full, 0)
        assert np.array_equal(counts(path, depth), want), depth
        assert np.array_equal(counts(path, depth, line=10), want[10]), depth
