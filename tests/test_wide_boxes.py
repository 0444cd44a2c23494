"""The grid and codes of the four-wide tree's 8-bit boxes (csrc/wide_box.h),
compiled for the host, in exact arithmetic: the stored box holds the exact one,
also where a node has no thickness on an axis, and its planes stay within what
the walk's error bounds count on."""
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "wide_box.h"
#include <cstdio>
// intervals (lo, hi) of one node's four children, as float bits, a line a node
int main() {
    unsigned u[8];
    while (std::scanf("%x %x %x %x %x %x %x %x", u, u + 1, u + 2, u + 3, u + 4, u + 5, u + 6, u + 7) == 8) {
        float v[8], mn, mx, base = 0;
        for (int k = 0; k < 8; ++k) v[k] = ptb::__uint_as_float_hd(u[k]);
        mn = v[0]; mx = v[1];
        for (int c = 1; c < 4; ++c) { mn = fminf(mn, v[2 * c]); mx = fmaxf(mx, v[2 * c + 1]); }
        unsigned e = 0;
        const int holds = ptb::wide_frame(mn, mx, base, e);
        std::printf("%d %x %u", holds, ptb::__float_as_uint_hd(base), e);
        for (int c = 0; c < 4; ++c)
            std::printf(" %u %u", ptb::wide_code_lo(v[2 * c], base, ptb::wide_scale(e)),
                        ptb::wide_code_hi(v[2 * c + 1], base, ptb::wide_scale(e)));
        std::printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def boxes(tmp_path_factory):
    d = tmp_path_factory.mktemp("wide")
    (d / "boxes.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", str(d / "boxes.cpp"),
                    "-I", os.path.join(ROOT, "pathtracingtutorial_b200", "csrc"),
                    "-I", "/usr/local/cuda/include", "-o", str(d / "boxes")], check=True)

    def run(v):
        text = "\n".join(" ".join(f"{x:x}" for x in row) for row in v.astype(np.float32).view(np.uint32))
        out = subprocess.run([str(d / "boxes")], input=text, capture_output=True, text=True, check=True).stdout
        rows = [line.split() for line in out.splitlines()]
        assert len(rows) == len(v)
        return [(int(r[0]), np.array(int(r[1], 16), np.uint32).view(np.float32).item(), int(r[2]),
                 [int(x) for x in r[3:]]) for r in rows]
    return run


def _cases(name):
    rng = np.random.default_rng(5)
    n = 2000
    if name == "flat":          # no thickness, every child on the same plane
        at = np.concatenate([[1, -1, 1.5, 548.8, -548.8, 1e-3, 3e29, -1e30, 1e-20, 0, 1e-38, 1e-44, 2.0 ** -80],
                             rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-30, 29, n)])
        return np.repeat(at.astype(np.float32)[:, None], 8, 1)
    base = (rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-12, 12, n)).astype(np.float32)
    if name == "thin":          # a few spacings of the coordinate thick
        v = np.repeat(base[:, None], 8, 1)
        for k in range(8):
            for _ in range(4):
                step = rng.random(n) < 0.4
                v[step, k] = np.nextafter(v[step, k], np.float32(np.inf))
    elif name == "across":      # from one side of zero to the other, sizes far apart
        v = (rng.uniform(-1, 1, (n, 8)) * 10.0 ** rng.uniform(-12, 12, (n, 8))).astype(np.float32)
    else:                       # ordinary boxes, small against their coordinates or not
        v = (base[:, None] + np.abs(base)[:, None] * 10.0 ** rng.uniform(-6, 1, (n, 1))
             * rng.uniform(0, 1, (n, 8))).astype(np.float32)
    v = v.reshape(n, 4, 2)
    v.sort(2)
    return v.reshape(n, 8)


@pytest.mark.parametrize("name", ["flat", "thin", "across", "ordinary"])
def test_stored_boxes_hold_the_exact_ones(boxes, name):
    v = _cases(name)
    for row, (holds, base, e, codes) in zip(v, boxes(v)):
        assert holds
        scale = Fraction(2) ** (e - 127)
        plane = [Fraction(base) + (128 + c if c < 128 else 2 * c) * scale for c in codes]
        for c in range(4):
            assert plane[2 * c] <= Fraction(float(row[2 * c])), (row, base, e, codes)
            assert plane[2 * c + 1] >= Fraction(float(row[2 * c + 1])), (row, base, e, codes)
        # what the conservative test's error bound takes for the base and the offsets
        most = max(Fraction(float(np.abs(row).max())), Fraction(2) ** -80)
        assert abs(Fraction(base)) <= Fraction(24, 10) * most and 510 * scale <= Fraction(54, 10) * most
