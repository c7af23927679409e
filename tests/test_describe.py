"""CPU: a plan's description names the kernel that runs: run-time radices only where
no kernel of fixed radices is compiled for the size."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "goldilocks_gb300", "csrc")


def compiled():
    """Size -> radices of the four-lane kernels that run in the run-time-radix
    kernel's place."""
    out = {}
    for f in ("mixed17", "mixed35", "small"):
        src = open(os.path.join(CSRC, "gl_kern_%s_fwd.cu" % f)).read()
        for r in re.findall(r"ENTRY3\w?\((\d+), (\d+), (\d+), 4,", src):
            a, b, c = map(int, r)
            out[a * b * c] = "%dx%dx%d" % (a, b, c)
    return out


@pytest.mark.parametrize("n,want", [
    (15360, "col 128 (16x8x1, 4 lanes) + row 120 (15x8x1, 4 lanes)"),
    (61440, "col 256 (16x16x1, 4 lanes) + row 240 (16x15x1, 4 lanes)"),
    (1536, "full 1536 (16x16x6, 4 lanes)"),
    (257 * 16, "rader 257 (one kernel) then 16: full 16 (16x1x1, 64 lanes)"),
    (48, "full 48 (16x3x1, 4 lanes, run-time radices)"),
])
def test_pinned(gl, n, want):
    assert gl.strategy(n).describe().split(" | gpu: ")[1] == want


def test_all_lengths(gl):
    sizes = compiled()
    assert len(sizes) > 30
    for n in gl.divisors():
        if n == 1 or n > 1 << 24 or n % 257 == 0 or n % 65537 == 0:
            continue
        for part in gl.strategy(n).describe().split(" | gpu: ")[1].split(" + "):
            m = int(part.split()[1])
            if "run-time radices" in part:
                assert m not in sizes, (n, part)
            elif m in sizes and "4 lanes)" in part and m & (m - 1):
                assert sizes[m] in part, (n, part)
