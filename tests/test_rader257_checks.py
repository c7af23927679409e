"""CPU: the index checks of a debug build (-DGL_DEVICE_CHECKS) in the one-kernel
Rader step over 257: clean on the true extents, set where a word lies outside."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, rand_field
from test_rader257 import HARNESS

CHECKED = HARNESS + r"""
extern "C" uint32_t emu_rader257_checked(int lanes, const uint64_t *src, uint64_t *dst, uint64_t L, uint64_t C,
                                         const uint32_t *index, const uint64_t *words, uint64_t in, uint64_t out) {
  uint32_t err = 0;
  const gl_rader257_args a{src, dst, L, C, index, index, words, words, words, words, words, in, out, &err};
  if (lanes == 8) run<8>(a);
  else run<16>(a);
  return err;
}
"""


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    d = tmp_path_factory.mktemp("rader257c")
    (d / "r.cpp").write_text(CHECKED)
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared", "-pthread", "-DGL_DEVICE_CHECKS",
                    "-I" + os.path.join(ROOT, "goldilocks_gb300", "csrc"), "-I" + os.path.join(ROOT, "tests"),
                    str(d / "r.cpp"), "-o", str(d / "r.so")], check=True)
    f = ctypes.CDLL(str(d / "r.so")).emu_rader257_checked
    f.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 2 + [ctypes.c_uint64] * 2 + [ctypes.c_void_p] * 2 + [ctypes.c_uint64] * 2
    f.restype = ctypes.c_uint32
    return f


@pytest.mark.parametrize("m,C", [(1, 1), (17, 1), (2, 16), (1, 20)])
@pytest.mark.parametrize("lanes", [8, 16])
def test_extents(emu, m, C, lanes):
    words = 257 * m * C
    index = np.array([pow(3, p, 257) for p in range(256)], dtype=np.uint32)
    table = rand_field(4096, seed=3)  # any words: only the indices are looked at
    src, guard = rand_field(words, seed=words), 64

    def run(lost_in, lost_out):
        dst = np.full(words + guard, 0x5555, dtype=np.uint64)
        bits = emu(lanes, src.ctypes.data, dst.ctypes.data, m * C, C, index.ctypes.data, table.ctypes.data,
                   words - lost_in, words - lost_out)
        assert (dst[words - lost_out:] == 0x5555).all()  # a checked store outside is skipped
        assert (dst[:words - lost_out] != 0x5555).all()
        return bits

    assert run(0, 0) == 0
    assert run(1, 0) == 1
    assert run(0, 1) == 2
    assert run(1, 1) == 3
