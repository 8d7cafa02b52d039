"""Two pixels a lane (large deep Mandelbrot frames) against one pixel a lane
(the frame schedule): the same counts and |z|^2, bit for bit, on views whose
deltas rescale often, leave the deep part, rebase and escalate, with an odd
number of pixels, and with depths that end inside a block."""
import numpy as np
import pytest

from mdz_gb300 import MpVal, parse_number
from mdz_gb300.stream import load_pool

pytestmark = pytest.mark.gpu

POOL = [c for c in load_pool() if c["fractal"] == 0]
# centre (None: c = i), log2 width, W, H, depth
CASES = [(None, -300, 641, 401, 997), (None, -180, 600, 403, 3001), (0, -250, 641, 379, 11003),
         (1, -700, 577, 421, 10502), (2, -165, 640, 400, 10999)]


@pytest.mark.parametrize("centre,zoom,W,H,depth", CASES)
def test_pairs_equal_single(renderer, monkeypatch, centre, zoom, W, H, depth):
    assert W * H > 64 * 24 * 152
    prec = 64 - zoom
    c = POOL[centre] if centre is not None else {"cx": "0", "cy": "1"}
    v = [MpVal.from_fraction(parse_number(x), prec) for x in (c["cx"], c["cy"], f"0x1p{zoom}")]
    got, mag, st = renderer.render_perturb(W, H, depth, *v, prec, want_mag=True)
    monkeypatch.setenv("MDZGPU_PERTURB", "frame")
    want, mag1, st1 = renderer.render_perturb(W, H, depth, *v, prec, want_mag=True)
    assert np.array_equal(got, want)
    assert np.array_equal(mag, mag1)
    assert all(st[k] == st1[k] for k in ("pixel_iters", "rebases", "escalated_fp64",
                                         "escalated_mp"))
