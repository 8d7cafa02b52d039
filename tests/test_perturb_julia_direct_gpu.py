"""Julia views of the burning ship formula whose FP64 pass loses its error
estimate and iterates the rest of a pixel directly, z' = f(z) + c with
the Julia constant.  The views are centred away from 0, where the first step of
the view's orbit is not the constant, and have attracting cycles, so that every
pixel is resolved: the counts are the multi-limb method's, but for the 0.1% of
the pixels (at least 2) that the other Julia views are allowed."""
import numpy as np
import pytest

from mdz_gb300 import MpVal, parse_number
from mdz_gb300.serve import RenderRequest, Server
from mdz_gb300.stream import load_pool

pytestmark = pytest.mark.gpu

POOL = load_pool()
OFF = {"cx": "0x1p-3", "cy": "-0x1p-4"}


@pytest.fixture(scope="module")
def server():
    with Server(0, arena_bytes=1 << 30) as s:
        yield s


# pool entry that is the Julia constant, centre (None: the same), log2 width
@pytest.mark.parametrize("pool,centre,zoom", [
    (3, OFF, -2), (3, OFF, -20), (3, None, -60), (4, OFF, -60), (4, None, -20)])
def test_direct_pixels_take_the_julia_constant(renderer, server, pool, centre, zoom):
    prec, W, H, depth, fractal = 264, 64, 48, 12000, 1
    val = lambda v: MpVal.from_fraction(parse_number(v), prec)
    c = [x for x in POOL if x["fractal"] == fractal][pool]
    at = centre or c
    julia = val(c["cx"]), val(c["cy"])
    view = val(at["cx"]), val(at["cy"]), val(f"0x1p{zoom}")
    got, _, st = renderer.render_perturb(W, H, depth, *view, prec, fractal=fractal, julia=julia)
    assert st["escalated_fp64"] - st["escalated_mp"] > 500
    q = RenderRequest(W, H, depth, *view, prec, fractal=fractal, method="multi_limb", family=1,
                      julia=julia)
    rid = server.submit(q)
    assert server.wait(rid)["state"] == "done"
    server.release(rid)
    assert int((got != q.counts).sum()) <= max(2, 0.001 * got.size)
