"""Timed cases: what a user of this renderer has it do, through its public calls.

A case names a method and a view (centre, span, formula, size, maximum
iterations); prepare() builds the view's exact numbers and the output
buffers, run() makes the one call a program makes per frame.  Another seed
pans the view by a fraction of its span, as moving through a zoom does.
Centres come from the repository's seeded views and from the serving
stream's pool of boundary points.

One Renderer (and one Server) serves all cases of a process, as in a program
that renders frame after frame.
"""
from __future__ import annotations

import math
import random
from fractions import Fraction

import numpy as np
import torch

from mdz_gb300 import MpVal, Renderer, parse_number
from mdz_gb300.cases import VIEWS
from mdz_gb300.serve import RenderRequest, Server
from mdz_gb300.stream import load_pool

_shared: dict = {}


def _renderer() -> Renderer:
    if "renderer" not in _shared:
        _shared["renderer"] = Renderer(0)
    return _shared["renderer"]


def _server() -> Server:
    if "server" not in _shared:
        _shared["server"] = Server(0, arena_bytes=2 << 30)
    return _shared["server"]


# Where the views look: (formula, centre x, centre y, share of the maximum
# iteration count an average pixel runs for).  Formula numbers as MDZ's:
# 0 Mandelbrot, 1 burning ship, 2 generalized celtic, 3 the hybrid.
def _centres() -> dict:
    if "centres" not in _shared:
        pool = load_pool()
        ship = [c for c in pool if c["fractal"] == 1]
        celtic = [c for c in pool if c["fractal"] == 2]
        mandel = [c for c in pool if c["fractal"] == 0]
        _shared["centres"] = {
            "whole": (0, "-0.75", "0", 0.229),
            "ship_whole": (1, "-0.45", "-0.5", 0.24),
            "celtic_whole": (2, "-0.5", "0.2", 0.22),
            "hybrid_whole": (3, "-0.6", "0.15", 0.20),
            "julia_whole": (0, "0", "0", 0.046),
            "c2": (0, VIEWS["c2"]["cx"], VIEWS["c2"]["cy"], 0.53),
            "c4": (0, VIEWS["c4"]["cx"], VIEWS["c4"]["cy"], 1.0),
            "i": (0, "0", "1", 0.42),
            "mandel": (0, mandel[0]["cx"], mandel[0]["cy"], 0.6),
            "ship": (1, ship[0]["cx"], ship[0]["cy"], 0.6),
            "celtic": (2, celtic[0]["cx"], celtic[0]["cy"], 0.6),
            # on the boundary of the basilica Julia set (c = -1), to 2^-264
            "basilica": (0, "0x3eb39f4eaddcc60ef5982f1b7617d2ba6fc62301a5894639d49988c9b3b1a228c3p-263",
                         "0xbc1addec0996522ce0c88d526247782f4f526904f09bd2ad7dcc9a5d1b14e67a49p-266", 0.37),
        }
    return _shared["centres"]


def listed() -> list[dict]:
    return [
        # the first picture a viewer shows: the whole set in a small window
        dict(name="fp64_preview", path="fp64", at="whole", W=240, H=180, span="3.0", depth=1000),
        # hardware-float zoom at the end of double precision, deep iteration
        dict(name="fp64_zoom", path="fp64", at="c2", W=960, H=540, span="1e-11", depth=20000),
        # an exported picture: Julia set, 3x3 supersampled, coloured on the GPU
        dict(name="image_julia_aa3", path="image", at="julia_whole", W=2877, H=1623, aa=3,
             span="3.2", depth=1000, julia="-0.8,0.156", interpolate=True),
        # multi-limb at MDZ's default 80 bits, where doubles run out
        dict(name="mp80", path="mp", at="c2", W=320, H=240, span="1e-13", depth=15000, bits=80),
        # multi-limb at 256 bits
        dict(name="mp256", path="mp", at="mandel", W=320, H=240, span="0x1p-200", depth=12000,
             bits=256),
        # multi-limb at 1088 bits, a small odd-sized window
        dict(name="mp1088", path="mp", at="mandel", W=201, H=151, span="0x1p-1000", depth=11000,
             bits=1088),
        # beyond one thread's registers: 2176 bits, a small exact check render
        dict(name="mp2176", path="mp", at="i", W=96, H=64, span="0x1p-2100", depth=4000,
             bits=2176),
        # the deep zoom: full HD at 2^-1000
        dict(name="perturb_deep", path="perturb", at="c4", W=1920, H=1080, span="0x1p-1000",
             depth=200000, bits=1088),
        # a moderate zoom on a boundary point, with pixels that need more
        # precision than the first pass has
        dict(name="perturb_mid", path="perturb", at="mandel", W=640, H=480, span="0x1p-100",
             depth=15000, bits=164),
        # burning ship around a boundary point
        dict(name="perturb_ship", path="perturb", at="ship", W=480, H=270, span="0x1p-300",
             depth=10000, bits=364),
        # a small Julia view with |z|^2 for smooth colouring
        dict(name="perturb_julia_small", path="perturb", at="basilica", W=161, H=121,
             span="0x1p-200", depth=3000, bits=264, julia="-1,0", mag=True),
        # a server's mix of requests of several sizes, depths and formulas
        dict(name="serve_mix", path="serve", requests=8, depth=16000),
    ]


def _log_uniform(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    """A case of the same paths at other sizes, depths, precisions and formulas."""
    most = {"fp64": 1e10, "image": 2.5e9, "mp": 6e11, "perturb": 5e10, "c4": 6e12}
    while True:
        path = rng.choice(["fp64", "image", "mp", "mp", "perturb", "perturb", "serve"])
        if path == "serve":
            return dict(path=path, requests=rng.randint(3, 9), depth=_log_uniform(rng, 11000, 20000))
        W = _log_uniform(rng, 64, 1920)
        H = max(16, int(W * rng.uniform(0.4, 1.1)))
        c = dict(path=path, W=W, H=H)
        if path == "fp64":
            at = rng.choice(["whole", "ship_whole", "celtic_whole", "hybrid_whole", "c2"])
            c.update(at=at, depth=_log_uniform(rng, 200, 20000),
                     span="%.6g" % (10 ** rng.uniform(-11, -2)) if at == "c2" else "3.1")
        elif path == "image":
            aa = rng.randint(1, 4)
            c.update(at=rng.choice(["julia_whole", "whole", "celtic_whole"]), aa=aa,
                     depth=_log_uniform(rng, 200, 2000), span="3.2",
                     interpolate=rng.random() < 0.5)
            c["W"], c["H"] = c["W"] * aa, c["H"] * aa
            if c["at"] == "julia_whole":
                c["julia"] = "-0.8,0.156"
        elif path == "mp":
            zoom = _log_uniform(rng, 30, 1500)
            at = rng.choice(["mandel", "ship", "celtic", "i"]) if zoom <= 1000 else "i"
            c.update(at=at, span="0x1p-%d" % zoom, bits=zoom + 50,
                     depth=_log_uniform(rng, 3000 if at == "i" else 10500, 15000))
        else:
            zoom = _log_uniform(rng, 40, 1000)
            at = rng.choice(["mandel", "i", "c4", "ship", "celtic", "basilica"])
            zoom = min(zoom, 200) if at == "basilica" else zoom
            # the centres' escape counts are near 10^4 (c4: 2 10^5)
            lo, hi = {"i": (2000, 20000), "basilica": (1000, 6000),
                      "c4": (200000, 200000)}.get(at, (10500, 20000))
            c.update(at=at, span="0x1p-%d" % zoom, bits=zoom + 64, mag=rng.random() < 0.3,
                     depth=_log_uniform(rng, lo, hi))
            if at == "basilica":
                c["julia"] = "-1,0"
        if work(c)["flops"] <= most.get(c["at"], most[path]):
            return c


def _mp_words(bits: int) -> int:
    return 2 * -(-(bits + 8 + 24) // 64)


def work(case: dict) -> dict:
    """The counts (and colours) once, and the iterations' arithmetic."""
    if case["path"] == "serve":
        n = sum(r["W"] * r["H"] for r in _serve_items(case, 0))
        return {"bytes": 4.0 * n, "flops": 16.0 * 0.4 * n * case["depth"]}
    n = case["W"] * case["H"]
    its = _centres()[case["at"]][3] * n * case["depth"]
    if case["path"] == "mp":
        w = _mp_words(case["bits"])
        # one product and two squares, truncated to the upper half, as
        # 32-bit multiply-adds; about ten additions of w words
        return {"bytes": 4.0 * n, "flops": its * (2.0 * w * w + 10.0 * w)}
    if case["path"] == "fp64":
        return {"bytes": 4.0 * n, "flops": 8.0 * its}
    if case["path"] == "image":
        return {"bytes": 8.0 * n + 4.0 * n / case["aa"] ** 2, "flops": 8.0 * its}
    return {"bytes": (8.0 if case.get("mag") else 4.0) * n, "flops": 16.0 * its}


def _pan(seed: int, span: Fraction, k: int = 0) -> tuple[Fraction, Fraction]:
    rng = random.Random(1000003 * seed + k)
    return tuple(Fraction(rng.randint(-65536, 65536), 1 << 20) * span for _ in range(2))


def _view(case: dict, seed: int) -> tuple:
    fractal, cx, cy, _ = _centres()[case["at"]]
    span = parse_number(case["span"])
    px, py = _pan(seed, span)
    return fractal, parse_number(cx) + px, parse_number(cy) + py, span


def _serve_items(case: dict, seed: int) -> list[dict]:
    """The mix: sizes, spans and formulas as the serving stream draws them,
    from the case alone; the seed pans each view."""
    rng = random.Random(17 * case["requests"] + case["depth"])
    items = []
    for k in range(case["requests"]):
        W, H = rng.choice([(240, 180), (320, 240), (640, 480)])
        at = rng.choice(["mandel"] * 7 + ["ship"] * 2 + ["celtic"])
        zoom = rng.randint(10, 1000)
        fractal, cx, cy, _ = _centres()[at]
        span = Fraction(1, 2 ** zoom)
        px, py = _pan(seed, span, k + 1)
        items.append(dict(W=W, H=H, fractal=fractal, cx=parse_number(cx) + px,
                          cy=parse_number(cy) + py, span=span, bits=zoom + 64,
                          depth=case["depth"] if k == 0 else _log_uniform(rng, 1000, case["depth"])))
    return items


def prepare(case: dict, seed: int) -> dict:
    s: dict = {"case": case}
    if case["path"] == "serve":
        s["server"] = _server()
        s["requests"] = [
            RenderRequest(r["W"], r["H"], r["depth"], MpVal.from_fraction(r["cx"], r["bits"]),
                          MpVal.from_fraction(r["cy"], r["bits"]),
                          MpVal.from_fraction(r["span"], r["bits"]), r["bits"],
                          fractal=r["fractal"], counts=np.zeros((r["H"], r["W"]), np.int32))
            for r in _serve_items(case, seed)]
        return s
    s["r"] = _renderer()
    fractal, cx, cy, span = _view(case, seed)
    W, H = case["W"], case["H"]
    s["fractal"], s["family"] = fractal, 1 if case.get("julia") else 0
    bits = case.get("bits", 53)
    julia = tuple(parse_number(v) for v in case["julia"].split(",")) if case.get("julia") else None
    top = cy + span * H / W / 2
    if case["path"] in ("fp64", "image"):
        s["rect"] = (float(cx - span / 2), float(cx + span / 2), float(top))
        s["julia"] = tuple(float(v) for v in julia) if julia else (0.0, 0.0)
    elif case["path"] == "mp":
        s["rect"] = tuple(MpVal.from_fraction(v, bits) for v in (cx - span / 2, top, span))
    else:
        s["view"] = tuple(MpVal.from_fraction(v, bits) for v in (cx, cy, span))
        s["julia"] = tuple(MpVal.from_fraction(v, bits) for v in julia) if julia else None
        s["mag"] = np.zeros((H, W), np.float32) if case.get("mag") else None
    if case["path"] == "image":
        aa = case["aa"]
        s["counts"] = torch.zeros((H, W), dtype=torch.int32, device="cuda")
        s["rgb"] = torch.zeros((H // aa, W // aa), dtype=torch.int32, device="cuda")
        rng = random.Random(seed)
        s["palette"] = np.array([rng.getrandbits(24) for _ in range(256)], np.uint32)
    else:
        s["out"] = np.zeros((H, W), np.int32)
    return s


def run(s: dict):
    case = s["case"]
    if case["path"] == "serve":
        srv = s["server"]
        ids = [srv.submit(q) for q in s["requests"]]
        for i in ids:
            srv.wait(i)
            srv.release(i)
        return [q.counts for q in s["requests"]]
    r, W, H, depth = s["r"], case["W"], case["H"], case["depth"]
    if case["path"] == "fp64":
        return r.render_fp64(W, H, depth, *s["rect"], family=s["family"], fractal=s["fractal"],
                             julia=s["julia"], out=s["out"])[0]
    if case["path"] == "image":
        r.render_fp64_device(W, H, depth, *s["rect"], s["counts"].data_ptr(), family=s["family"],
                             fractal=s["fractal"], julia=s["julia"])
        r.colour_device(s["counts"].data_ptr(), W, H, case["aa"], s["palette"],
                        s["rgb"].data_ptr(), colour_scale=1.37, interpolate=case["interpolate"],
                        offset=3)
        return [s["counts"], s["rgb"]]
    if case["path"] == "mp":
        return r.render_mp(W, H, depth, *s["rect"], case["bits"], fractal=s["fractal"],
                           out=s["out"])[0]
    counts, mag, _ = r.render_perturb(W, H, depth, *s["view"], case["bits"],
                                      want_mag=s["mag"] is not None, out=s["out"], mag=s["mag"],
                                      fractal=s["fractal"], julia=s["julia"])
    return [counts] if mag is None else [counts, mag]


def exact(case: dict, seed: int):
    """The outputs are iteration counts and packed colours (whole numbers),
    and |z|^2 of orbits that 64-bit arithmetic cannot follow."""
    return None
