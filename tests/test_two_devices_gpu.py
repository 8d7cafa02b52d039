"""Multi-limb frames on a second GPU after a first one in the same process: a
frame kernel of 20 words or more needs each device's leave for its shared
memory.  Needs two GPUs."""
from fractions import Fraction

import numpy as np
import pytest

from mdz_gb300 import MpVal, Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", [16, 20, 36])
def test_frame_on_each_device(words):
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("one GPU")
    prec = 32 * words - 8
    rect = [MpVal.from_fraction(Fraction(v), prec) for v in ("-9/4", "5/4", "3")]
    frames = []
    for device in (0, 1, 0):
        with Renderer(device) as r:
            frames.append(r.render_mp(61, 37, 300, *rect, prec, words=words)[0].copy())
    assert len(np.unique(frames[0])) > 10
    assert all(np.array_equal(f, frames[0]) for f in frames[1:])
