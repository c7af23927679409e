"""CPU: the uniform form of a column pass (one column index per tile: tables of
the tile for the pass twiddle and the coset factor) against the general form,
both from the kernel source on the emulator, over what the launcher lets it
take: two and three rounds, both directions, with and without a coset factor,
zero padding, a first column other than zero and a scaled twiddle table."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import P, ROOT, rand_field
from test_kernel_emulation import F_IN_TW, F_LOAD_LF, F_PASS_TW, F_STORE_LF, NOLIM, root, table

HARNESS = r"""
#include "kernel_emu.cpp"
template <int R1, int R2, int R3, int LANES, int NT, bool INV, bool UNI>
static void run_tiles(const gl_pass_args &a) {
  for (unsigned x = 0; x < a.lanes / LANES; x++) {
    memset(sm, 0xA5, sizeof(sm));
    std::barrier<> bar(NT);
    g_bar = &bar;
    std::vector<std::thread> th;
    for (int t = 0; t < NT; t++)
      th.emplace_back([&a, t, x] {
        threadIdx.x = t;
        gl_block3<R1, R2, R3, LANES, NT, INV, false, UNI>(a, x, 0, 0, sm);
      });
    for (auto &t : th) t.join();
  }
}
extern "C" int emu_uniform(int r1, int r2, int r3, int inv, int uni, const uint64_t *in, uint64_t *out, int64_t stride,
                           uint32_t lanes, uint32_t flags, const uint64_t *tw_m, const uint64_t *lo, const uint64_t *hi,
                           uint32_t div, uint32_t limit, const uint64_t *ilo, const uint64_t *ihi, uint64_t jmul,
                           uint64_t col0, uint64_t unscale, uint64_t words) {
  gl_pass_args a{};
  a.in = in; a.out = out; a.in_ls = a.out_ls = 1; a.in_is = a.out_is = stride;
  a.lanes = lanes; a.flags = flags; a.tw_m = a.tw_r2 = tw_m; a.tw_lo = lo; a.tw_hi = hi; a.tw_lane_div = div;
  a.in_limit = limit; a.itw_lo = ilo; a.itw_hi = ihi; a.itw_jmul = jmul; a.tw_col0 = col0; a.tw_unscale = unscale;
  a.dbg_in_words = a.dbg_out_words = words; a.dbg_err = &g_dbg_err;
#define SHAPE_U(R1, R2, R3, LN, NT)                                         \
  if (r1 == R1 && r2 == R2 && r3 == R3) {                                   \
    if (inv && uni) run_tiles<R1, R2, R3, LN, NT, true, true>(a);            \
    else if (inv) run_tiles<R1, R2, R3, LN, NT, true, false>(a);             \
    else if (uni) run_tiles<R1, R2, R3, LN, NT, false, true>(a);             \
    else run_tiles<R1, R2, R3, LN, NT, false, false>(a);                     \
    return 0;                                                               \
  }
  SHAPE_U(8, 8, 8, 8, 512)
  SHAPE_U(16, 16, 1, 16, 256)
  SHAPE_U(16, 8, 1, 32, 256)
  SHAPE_U(8, 8, 1, 32, 256)
  return -1;
}
"""


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    d = tmp_path_factory.mktemp("uniform")
    (d / "u.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared", "-pthread", "-DGL_DEVICE_CHECKS",
                    "-I" + os.path.join(ROOT, "goldilocks_gb300", "csrc"), "-I" + os.path.join(ROOT, "tests"),
                    str(d / "u.cpp"), "-o", str(d / "u.so")], check=True)
    lib = ctypes.CDLL(str(d / "u.so"))
    vp, i64, u32, u64 = ctypes.c_void_p, ctypes.c_int64, ctypes.c_uint32, ctypes.c_uint64
    lib.emu_uniform.argtypes = [ctypes.c_int] * 5 + [vp, vp, i64, u32, u32, vp, vp, vp, u32, u32, vp, vp] + [u64] * 4
    lib.emu_check_flags.restype = u32
    return lib


@pytest.mark.parametrize("shape,lanes", [((8, 8, 8), 8), ((16, 16, 1), 16), ((16, 8, 1), 32), ((8, 8, 1), 32)])
@pytest.mark.parametrize("inv", [False, True])
@pytest.mark.parametrize("coset,limit,col0", [(False, NOLIM, 0), (True, NOLIM, 0), (True, 40, 0), (False, NOLIM, 3)])
def test_uniform_equals_general(emu, shape, lanes, inv, coset, limit, col0):
    m = shape[0] * shape[1] * shape[2]
    n2, C = 2, 2 * lanes  # two column indices, two tiles each
    n, cols = m * 8, n2 * C
    w = root(n, inv)
    scale = pow(n, P - 2, P) if inv else 1
    lo, hi = table(w, 4096, scale), table(pow(w, 4096, P), (n + 4095) // 4096)
    # the coset factor's tables end with the last index that is not padded
    last = min(limit, m) * n2
    ilo, ihi = table(7, min(4096, last)), table(pow(7, 4096, P), (last + 4095) // 4096)
    x = rand_field(m * cols, seed=m + inv)
    x[:8] = 2**64 - 1
    flags = F_PASS_TW | F_LOAD_LF | F_STORE_LF | (F_IN_TW if coset else 0)
    got = []
    for uni in (0, 1):
        out = np.zeros_like(x)
        tm = table(root(m, inv), m)
        assert emu.emu_uniform(*shape, int(inv), uni, x.ctypes.data, out.ctypes.data, cols, cols, flags,
                               tm.ctypes.data, lo.ctypes.data, hi.ctypes.data, C, limit, ilo.ctypes.data,
                               ihi.ctypes.data, n2, col0, (n * 2**64 % P) if inv else 0, m * cols) == 0
        assert emu.emu_check_flags() == 0
        got.append(out)
    assert np.array_equal(got[0], got[1])
