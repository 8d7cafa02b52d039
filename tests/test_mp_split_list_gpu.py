"""Escalation lists of a few to 64 pixels an SM, four warps for 32 pixels: the
pixels a perturbation render hands to the multi-limb pass get the counts and
|z|^2 the one-thread kernel gives the same pixels, at word counts that use that
kernel, with lists of several blocks an SM, of less than a pixel an SM, and of
lanes that end thousands of iterations apart."""
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal, parse_number, perturb_pixel_c
from mdz_gb300.stream import load_pool

pytestmark = pytest.mark.gpu

POOL = load_pool()


# formula, log2 width, precision, words, W, H, depth, pixels an SM
@pytest.mark.parametrize("fractal,zoom,prec,words,W,H,depth,most", [
    (2, -220, 284, 12, 97, 71, 10600, 32), (2, -200, 264, 10, 97, 70, 10600, 32),
    (1, -300, 364, 16, 33, 21, 10000, 1),
    (1, -300, 364, 16, 241, 179, 10000, 32), (1, -400, 464, 16, 1280, 720, 10300, 64),
    (2, -500, 564, 20, 160, 121, 10400, 32), (1, -600, 664, 24, 640, 361, 10600, 32),
    (1, -881, 945, 34, 640, 480, 16000, 64)])
def test_split_list_counts(renderer, fractal, zoom, prec, words, W, H, depth, most):
    c = [x for x in POOL if x["fractal"] == fractal][0]
    cx, cy, w = (MpVal.from_fraction(parse_number(v), prec)
                 for v in (c["cx"], c["cy"], f"0x1p{zoom}"))
    got, mag, st = renderer.render_perturb(W, H, depth, cx, cy, w, prec, want_mag=True,
                                           fractal=fractal)
    _, listed = renderer.last_escalations()
    assert len(listed) == st["escalated_mp"]
    if not len(listed):
        pytest.skip("no pixel of this view reaches the multi-limb pass")
    assert len(listed) <= most * 152
    # the one-thread kernel on the same pixels, one frame of one pixel each
    picks = sorted({0, len(listed) - 1, *range(0, len(listed), max(1, len(listed) // 8))})
    for pix in listed[picks]:
        line, ix = divmod(int(pix), W)
        x, y = perturb_pixel_c(cx, cy, w, W, H, ix, line)
        one, s1 = renderer.render_mp(1, 1, depth, MpVal.from_fraction(x, 32 * words - 8),
                                     MpVal.from_fraction(y, 32 * words - 8),
                                     MpVal.from_fraction(Fraction(1, 2 ** 40), 64),
                                     32 * words - 8, words=words, fractal=fractal)
        assert s1["words"] == words
        assert got[line, ix] == one[0, 0], (ix, line)
