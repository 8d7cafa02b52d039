"""Short escalation lists, one pixel a block: the pixels a perturbation render
hands to the multi-limb pass get the counts (and |z|^2) the one-thread kernel
gives the same pixels, at every word count the short-list kernel is used for."""
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal, parse_number, perturb_pixel_c
from mdz_gb300.stream import load_pool

pytestmark = pytest.mark.gpu

POOL = load_pool()


# formula, log2 width, precision, words, W, H, depth
@pytest.mark.parametrize("fractal,zoom,prec,words,W,H,depth", [
    (1, -300, 364, 16, 48, 37, 10400), (2, -500, 564, 20, 40, 31, 10400),
    (1, -600, 664, 24, 41, 30, 10400), (2, -700, 764, 28, 40, 30, 10400),
    (1, -881, 945, 34, 48, 36, 10600), (1, -1000, 1090, 36, 48, 36, 10600)])
def test_short_list_counts(renderer, fractal, zoom, prec, words, W, H, depth):
    c = [x for x in POOL if x["fractal"] == fractal][0]
    cx, cy, w = (MpVal.from_fraction(parse_number(v), prec)
                 for v in (c["cx"], c["cy"], f"0x1p{zoom}"))
    got, mag, st = renderer.render_perturb(W, H, depth, cx, cy, w, prec, want_mag=True,
                                           fractal=fractal)
    _, listed = renderer.last_escalations()
    assert len(listed) == st["escalated_mp"]
    if not len(listed):
        pytest.skip("no pixel of this view reaches the multi-limb pass")
    # the one-thread kernel on the same pixels, one frame of one pixel each
    for pix in listed[:: max(1, len(listed) // 6)]:
        line, ix = divmod(int(pix), W)
        x, y = perturb_pixel_c(cx, cy, w, W, H, ix, line)
        one, s1 = renderer.render_mp(1, 1, depth, MpVal.from_fraction(x, 32 * words - 8),
                                     MpVal.from_fraction(y, 32 * words - 8),
                                     MpVal.from_fraction(Fraction(1, 2 ** 40), 64),
                                     32 * words - 8, words=words, fractal=fractal)
        assert s1["words"] == words
        assert got[line, ix] == one[0, 0], (ix, line)
