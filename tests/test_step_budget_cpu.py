"""The iterations a pixel may take in one step of a perturbation frame are about
8 ms of the kernel that takes this step: two pixels a lane while enough are
left, one a lane for the rest of the same frame."""
import subprocess
from pathlib import Path

import pytest

from mdz_gb300 import build

ROOT = Path(__file__).resolve().parents[1]
SMS = 152
PAIRS = 64 * 24 * SMS    # pixels from which on a step takes two a lane

SRC = r"""
#include "internal.h"
int main()
{
    mdz::PerturbLaunch p;
    const unsigned att = 0;
    p.att = &att;
    int fractal, hs_e;
    unsigned left;
    while (scanf("%d %d %u", &fractal, &hs_e, &left) == 3) {
        p.fractal = fractal;
        p.hs_e = hs_e;
        printf("%u\n", mdz::step_budget(SMS, p, left));
    }
}
"""


@pytest.fixture(scope="module")
def budgets(tmp_path_factory):
    d = tmp_path_factory.mktemp("budget")
    src, exe = d / "budget.cu", d / "budget"
    src.write_text(SRC.replace("SMS", str(SMS)))
    subprocess.run([build.nvcc(), "-std=c++17", "-I", str(build.CSRC), str(src), "-o", str(exe)],
                   check=True)

    def run(rows):
        text = "\n".join(" ".join(str(v) for v in r) for r in rows)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True)
        return [int(v) for v in out.stdout.split()]
    return run


def test_budget_follows_the_pixels_left(budgets):
    rows, want = [], []
    for fractal, hs_e in ((0, -1010), (0, -160), (1, -1010), (2, -1010)):
        for left in (1, 1000, PAIRS - 1, PAIRS, 2 * PAIRS, 1920 * 1080, 10 ** 8):
            pairs = fractal == 0 and hs_e < -160 and left >= PAIRS
            b = (1.5e12 if pairs else 3e11) * 8e-3 / left
            rows.append((fractal, hs_e, left))
            want.append(int(min(max(b, 256.0), 2.0 ** 24)) & ~3)
    assert budgets(rows) == want
