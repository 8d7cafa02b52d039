"""The FP64 kernel where its products leave the integer path, its orbits
repeat, or its tiles are ragged: bit-exact against the CPU oracle's double
loops."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# W, H, depth, xmin, xmax, ymax, family, julia
CASES = {
    # rows on the real axis: wim stays 0
    "real_axis": (65, 9, 700, -2.0, 0.5, 0.15384615384615385, 0, (0.0, 0.0)),
    # exact cycles 0 -> -1 -> 0 and 0 -> 0, and orbits that reach them
    "cycle2": (64, 64, 5000, -1.25, -0.75, 0.25, 0, (0.0, 0.0)),
    # z decays through the denormals to 0; c = 0
    "julia0": (33, 31, 3000, -1.2, 1.2, 1.1, 1, (0.0, 0.0)),
    # c_im = 0: wim alone decays through the denormals
    "julia_real": (40, 23, 3000, -1.5, 1.5, 0.8, 1, (-0.5, 0.0)),
    # denormal, tiny and huge coordinates
    "denormal": (9, 5, 50, -1e-310, 1e-310, 1e-310, 0, (0.0, 0.0)),
    "tiny_julia": (17, 9, 400, -1e-160, 1e-160, 1e-155, 1, (-0.1, 1e-300)),
    "huge": (16, 8, 20, -1e200, 1e200, 1e200, 0, (0.0, 0.0)),
    "overflow": (8, 8, 20, -1e308, 1e307, 1e308, 1, (1e308, -1e308)),
    "wide": (31, 17, 60, -40.0, 40.0, 20.0, 0, (0.0, 0.0)),
    # one pixel, one row, one column, one iteration
    "one": (1, 1, 500, -0.1, 0.1, 0.0, 0, (0.0, 0.0)),
    "row": (301, 1, 300, -2.0, 0.6, 0.3, 0, (0.0, 0.0)),
    "column": (1, 301, 300, -0.7, -0.69, 1.2, 0, (0.0, 0.0)),
    "depth1": (19, 7, 1, -2.0, 2.0, 1.0, 0, (0.0, 0.0)),
    "depth2": (19, 7, 2, -2.0, 2.0, 1.0, 0, (0.0, 0.0)),
}


@pytest.mark.parametrize("fractal", [0, 1, 2, 3])
@pytest.mark.parametrize("name", sorted(CASES))
def test_fp64_edges(renderer, name, fractal):
    W, H, depth, xmin, xmax, ymax, family, julia = CASES[name]
    got, st = renderer.render_fp64(W, H, depth, xmin, xmax, ymax, family, fractal, julia)
    want, its = O.render_fp64(W, H, depth, xmin, xmax, ymax, family, fractal, julia)
    assert np.array_equal(got, want)
    assert st["pixel_iters"] == its
