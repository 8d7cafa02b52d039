"""Rows on the real axis (z_0 and c real), whose pixels take a step of their own,
against the CPU oracle: every formula, both families, a row in the middle of
tiles, at a tile's edge and alone, +0 and -0, escapes at once and late, cycles,
orbits that end in zero, overflow, infinities and NaN, and coordinates below
the normal range."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

# xmin, xmax, ymax, W, H: the axis in row ymax W / (xmax - xmin)
VIEWS = [(-2.25, 0.75, 1.125, 96, 72), (-2.0, 2.0, 0.0, 65, 1), (-2.0, 2.0, -0.0, 33, 9),
         (0.0, 0.25, 0.125, 64, 33), (-2.0 ** 40, 2.0 ** 40, 2.0 ** 38, 64, 12),
         (-1e200, 1e200, 0.0, 32, 3), (-np.inf, 1.0, 0.0, 24, 1), (0.0, np.inf, 0.0, 24, 1),
         (-1e-310, 1e-310, 0.0, 16, 2), (-1e-160, 1e-160, 0.0, 40, 5)]
JULIA = [(-1.0, 0.0), (0.25, -0.0), (0.0, 0.0), (-1.7548776662466927, 0.0), (-2.0, 0.0),
         (-0.75, 0.5)]


@pytest.mark.parametrize("fractal", [0, 1, 2, 3])
@pytest.mark.parametrize("depth", [1, 2, 3, 5, 1023])
def test_rows_on_the_axis(renderer, fractal, depth):
    for view in VIEWS:
        xmin, xmax, ymax, W, H = view
        for julia in [None] + JULIA:
            got, _ = renderer.render_fp64(W, H, depth, xmin, xmax, ymax,
                                          family=1 if julia else 0, fractal=fractal,
                                          julia=julia or (0.0, 0.0))
            want, _ = oracle.render_fp64(W, H, depth, xmin, xmax, ymax,
                                         family=1 if julia else 0, fractal=fractal,
                                         julia=julia or (0.0, 0.0))
            assert np.array_equal(got, want), (view, julia)
