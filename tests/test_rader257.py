"""CPU: the fused Rader step over 257 (kernel source on the host, one thread per
CUDA thread) against the oracle's 257-point transforms and the twiddle, for full
tiles, a last tile with lanes missing, one column and several, both directions."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import P, ROOT, rand_field
from test_kernel_emulation import root, table

HARNESS = r"""
#include "kernel_emu.cpp"
#include "gl_rader257.cuh"
template <int LN>
static void run(const gl_rader257_args &a) {
  for (uint64_t x = 0; x < (a.L + LN - 1) / LN; x++) {
    memset(sm, 0xA5, sizeof(sm));
    std::barrier<> bar(LN * 16);
    g_bar = &bar;
    std::vector<std::thread> th;
    for (int t = 0; t < LN * 16; t++)
      th.emplace_back([&a, t, x] { threadIdx.x = t; gl_rader257_block<LN>(a, x, sm); });
    for (auto &t : th) t.join();
  }
}
extern "C" void emu_rader257(int lanes, const uint64_t *src, uint64_t *dst, uint64_t L, uint64_t C, const uint32_t *gp,
                             const uint32_t *gn, const uint64_t *tf, const uint64_t *ti, const uint64_t *bhat,
                             const uint64_t *lo, const uint64_t *hi) {
  const gl_rader257_args a{src, dst, L, C, gp, gn, tf, ti, bhat, lo, hi};
  if (lanes == 8) run<8>(a);
  else run<16>(a);
}
"""


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    d = tmp_path_factory.mktemp("rader257")
    (d / "r.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared", "-pthread",
                    "-I" + os.path.join(ROOT, "goldilocks_gb300", "csrc"), "-I" + os.path.join(ROOT, "tests"),
                    str(d / "r.cpp"), "-o", str(d / "r.so")], check=True)
    lib = ctypes.CDLL(str(d / "r.so"))
    lib.emu_rader257.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 2 + [ctypes.c_uint64] * 2 + [ctypes.c_void_p] * 7
    return lib


@pytest.mark.parametrize("m,C", [(1, 1), (16, 1), (17, 1), (48, 1), (1, 3), (8, 3), (2, 16), (1, 20)])
@pytest.mark.parametrize("inv", [False, True])
@pytest.mark.parametrize("lanes", [8, 16])
def test_fused_step(emu, oracle, m, C, inv, lanes):
    n, L = 257 * m, m * C
    w = root(n, inv)
    gp = np.array([pow(3, p, 257) for p in range(256)], dtype=np.uint32)
    gn = np.array([pow(3, 256 - p, 257) for p in range(256)], dtype=np.uint32)
    wq = root(257, inv)
    bhat = oracle.ntt(np.array([pow(wq, int(s), P) for s in gn], dtype=np.uint64))
    scale = pow(257, P - 2, P) if inv else 1
    lo = np.array([scale * pow(w, e, P) % P for e in range(4096)], dtype=np.uint64)
    hi = np.array([pow(w, 4096 * e, P) for e in range((n + 4095) // 4096)], dtype=np.uint64)
    tf, ti = table(root(256), 256), table(root(256, True), 256, pow(256, P - 2, P))
    lo, hi, bhat = (np.array([int(v) * 2**64 % P for v in a], dtype=np.uint64) for a in (lo, hi, bhat))
    x = rand_field(257 * L, seed=L + inv)
    x[:2] = 2**64 - 1
    out = np.full_like(x, 0x5555)
    tables = (gp, gn, tf, ti, bhat, lo, hi)
    emu.emu_rader257(lanes, x.ctypes.data, out.ctypes.data, L, C, *(a.ctypes.data for a in tables))
    rows = x.reshape(257, L)
    for l in range(0, L, 5 if L > 8 else 1):
        y = (oracle.intt if inv else oracle.ntt)(rows[:, l] % np.uint64(P))
        j2, c = divmod(l, C)
        want = [int(v) * pow(w, j2 * k, P) % P for k, v in enumerate(y)]
        assert out.reshape(m, 257, C)[j2, :, c].tolist() == want, l
