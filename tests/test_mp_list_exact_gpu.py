"""The kernels of short multi-limb lists against the one-thread kernel, bit for
bit: every pixel a perturbation render hands to the multi-limb pass has the
count and |z|^2 that the server's multi-limb method (one thread a pixel, the
same coordinates and words) gives it.

Each case says which kernel is to take its list, and its length in pixels an SM
shows that it did: one pixel a block up to PIXEL, four warps for 32 pixels from
there up to SPLIT.  All formulas and the Julia family, pixels that escape and
pixels that do not, alone and with another render on the GPU."""
import json
import threading
from pathlib import Path

import numpy as np
import pytest

from mdz_gb300 import MpVal, Renderer, parse_number
from mdz_gb300.serve import RenderRequest, Server
from mdz_gb300.stream import load_pool

pytestmark = pytest.mark.gpu

GOLD = Path(__file__).resolve().parent / "golden"
POOL = load_pool()
HYBRID = json.loads((GOLD / "perturb_variant_views.json").read_text())["v_b_120"]
JULIA = json.loads((GOLD / "perturb_julia_views.json").read_text())

# pixels an SM, by words (split_list_per_sm, pixel_list_per_sm)
SPLIT = {10: 32, 12: 32, 16: 64, 20: 64, 24: 64, 28: 64, 34: 64, 36: 64}
PIXEL = {24: 3, 28: 6, 34: 8, 36: 12}

# kernel, view, log2 width, precision, words, W, H, depth
CASES = [
    ("split", "celtic", -200, 264, 10, 160, 120, 10600),
    ("split", "celtic", -220, 284, 12, 161, 119, 10600),
    ("split", "ship", -300, 364, 16, 64, 48, 10400),
    ("split", "mandelbrot", -200, 364, 16, 64, 48, 11000),
    ("split", "hybrid", -120, 364, 16, 160, 120, 12000),
    ("split", "julia", -200, 364, 16, 320, 240, 3000),
    ("split", "celtic", -500, 564, 20, 160, 120, 10600),
    ("split", "ship", -600, 664, 24, 320, 240, 10600),
    ("split", "hybrid", -120, 664, 24, 160, 120, 12000),
    ("split", "celtic", -700, 764, 28, 320, 240, 10600),
    ("split", "celtic", -881, 945, 34, 320, 240, 10600),
    ("split", "julia", -200, 945, 34, 320, 240, 3000),
    ("split", "celtic", -1000, 1090, 36, 320, 240, 10600),
    ("pixel", "ship", -600, 664, 24, 64, 48, 10400),
    ("pixel", "mandelbrot", -200, 664, 24, 64, 48, 11000),
    ("pixel", "julia", -200, 664, 24, 64, 48, 3000),
    ("pixel", "celtic", -700, 764, 28, 64, 48, 10600),
    ("pixel", "hybrid", -120, 945, 34, 160, 120, 12000),
    ("pixel", "ship-julia", -100, 945, 34, 64, 48, 4000),
    ("pixel", "ship", -1000, 1090, 36, 160, 120, 10600),
]
BESIDE = [CASES[4], CASES[10], CASES[17]]


def view_of(name):
    """formula, centre, Julia constant"""
    if name == "hybrid":
        return 3, (HYBRID["cx"], HYBRID["cy"]), None
    if name in ("julia", "ship-julia"):
        m = JULIA["j_basilica_200" if name == "julia" else "j_ship_100"]
        return m["fractal"], (m["cx"], m["cy"]), (m["julia_re"], m["julia_im"])
    fractal = ["mandelbrot", "ship", "celtic"].index(name)
    c = [x for x in POOL if x["fractal"] == fractal][0]
    return fractal, (c["cx"], c["cy"]), None


@pytest.fixture(scope="module")
def server():
    with Server(0, arena_bytes=1 << 30) as s:
        yield s


@pytest.fixture(scope="module")
def sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


def check(renderer, server, sms, kernel, view, zoom, prec, words, W, H, depth):
    fractal, centre, julia = view_of(view)
    val = lambda v: MpVal.from_fraction(parse_number(v), prec)
    cx, cy, w = val(centre[0]), val(centre[1]), val(f"0x1p{zoom}")
    j = tuple(val(v) for v in julia) if julia else None
    got, mag, st = renderer.render_perturb(W, H, depth, cx, cy, w, prec, want_mag=True,
                                           fractal=fractal, julia=j)
    _, listed = renderer.last_escalations()
    assert len(listed) == st["escalated_mp"] > 0
    low = 0 if kernel == "pixel" else PIXEL.get(words, 0) * sms
    high = (PIXEL if kernel == "pixel" else SPLIT)[words] * sms
    assert low < len(listed) <= high
    q = RenderRequest(W, H, depth, cx, cy, w, prec, fractal=fractal, method="multi_limb",
                      want_mag=True, family=1 if j else 0, julia=j)
    rid = server.submit(q)
    done = server.wait(rid)
    server.release(rid)
    assert done["state"] == "done" and done["words"] == words
    at = listed.astype(np.int64)
    assert np.array_equal(got.ravel()[at], q.counts.ravel()[at])
    assert np.array_equal(mag.ravel()[at], q.mag.ravel()[at])


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}{c[4]}-{c[1]}")
def test_list_equals_one_thread_kernel(renderer, server, sms, case):
    check(renderer, server, sms, *case)


@pytest.mark.parametrize("case", BESIDE, ids=lambda c: f"{c[0]}{c[4]}-{c[1]}")
def test_list_beside_another_render(renderer, server, sms, case):
    prec, stop = 248, threading.Event()
    val = lambda v: MpVal.from_fraction(parse_number(v), prec)
    rect = val("-2.25"), val("1.25"), val("3.0")

    def other():
        with Renderer(0) as r:
            while not stop.is_set():
                r.render_mp(640, 480, 2000, *rect, prec)

    t = threading.Thread(target=other)
    t.start()
    try:
        for _ in range(3):
            check(renderer, server, sms, *case)
    finally:
        stop.set()
        t.join()
