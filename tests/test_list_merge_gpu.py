"""The FP64 perturbation pass moves pixels between warps as its list runs out;
a pixel's count and |z|^2 must not depend on which others share the list.

A frame's middle rows, rendered as a frame of their own about the same centre,
have the same offsets and the same reference orbit, so they agree bit for bit.
Sizes: a list longer than all lanes of the GPU, one of a few warps an SM, one
of a few warps in all; a last tile that is not full in each."""
import numpy as np
import pytest

from mdz_gb300 import MpVal, parse_number
from mdz_gb300.stream import load_pool

pytestmark = pytest.mark.gpu

POOL = [c for c in load_pool() if c["fractal"] == 0]


@pytest.mark.parametrize("centre,zoom,W,heights,depth,julia", [
    (0, -100, 641, (479, 151, 33, 1), 11001, None),
    (1, -60, 333, (210, 40, 2), 12000, None),
    (None, -200, 163, (121, 21, 3), 2999, "-1"),
])
def test_rows_do_not_depend_on_the_frame(renderer, centre, zoom, W, heights, depth, julia):
    prec = 64 - zoom
    if centre is None:
        c = {"cx": "0x3eb39f4eaddcc60ef5982f1b7617d2ba6fc62301a5894639d49988c9b3b1a228c3p-263",
             "cy": "0xbc1addec0996522ce0c88d526247782f4f526904f09bd2ad7dcc9a5d1b14e67a49p-266"}
    else:
        c = POOL[centre]
    v = [MpVal.from_fraction(parse_number(x), prec) for x in (c["cx"], c["cy"], f"0x1p{zoom}")]
    j = (MpVal.from_fraction(parse_number(julia), prec),
         MpVal.from_fraction(parse_number("0"), prec)) if julia else None
    H = heights[0]
    full, fmag, st = renderer.render_perturb(W, H, depth, *v, prec, want_mag=True, julia=j)
    assert st["escalated_fp64"] > 0
    for h in heights[1:]:
        k = (H - h) // 2
        assert H - h == 2 * k
        part, mag, _ = renderer.render_perturb(W, h, depth, *v, prec, want_mag=True, julia=j)
        assert np.array_equal(part, full[k:k + h])
        assert np.array_equal(mag, fmag[k:k + h])
