"""CPU: the four-lane kernels of fixed radices against the run-time-radix kernel
whose launches they take over, both from the kernel source on the emulator, in
every form such a launch has: orders of load and store, a scaled first twiddle,
a pass twiddle from two tables or a full one, zero padding with a coset factor,
spectrum factors, pointer tables, and a last tile with lanes missing."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import P, ROOT, rand_field
from test_kernel_emulation import NOLIM, root, table

CSRC = os.path.join(ROOT, "goldilocks_gb300", "csrc")
PASS_TW, SCALE, LOAD_LF, STORE_LF, IN_TW, TW_TABLE, LOAD_CG, PTR, MUL, MONT = (1 << i for i in range(10))


def shapes():
    """Radices and threads of the compiled kernels (those in both directions' files
    are the same list)."""
    src = open(os.path.join(CSRC, "gl_kern_small_fwd.cu")).read()
    return [tuple(map(int, t)) for t in re.findall(r"ENTRY3M\((\d+), (\d+), (\d+), 4, (\d+),", src)]


HARNESS = r"""
#include "kernel_emu.cpp"
extern "C" int emu_fixed(int r1, int r2, int r3, int inv, int fixed, const uint64_t *in, uint64_t *out, uint64_t words,
                         int64_t ls, int64_t is, uint32_t lanes, uint32_t flags, const uint64_t *tw_m,
                         const uint64_t *tw_r2, const uint64_t *lo, const uint64_t *hi, const uint64_t *full,
                         int64_t ld, uint32_t div, uint32_t limit, const uint64_t *ilo, const uint64_t *ihi,
                         uint64_t jmul, uint64_t unscale, const uint64_t *mul, uint32_t items) {
  gl_pass_args a{};
  a.in = in; a.out = out; a.in_ls = a.out_ls = a.mul_ls = ls; a.in_is = a.out_is = is;
  a.in_bs = a.out_bs = a.mul_bs = (int64_t)(words / items);
  a.lanes = lanes; a.flags = flags; a.tw_m = tw_m; a.tw_r2 = tw_r2; a.tw_lo = lo; a.tw_hi = hi;
  a.tw_full = full; a.tw_ld = ld; a.tw_lane_div = div; a.in_limit = limit; a.itw_lo = ilo; a.itw_hi = ihi;
  a.itw_jmul = jmul; a.tw_unscale = unscale; a.mul = mul;
  a.dbg_in_words = a.dbg_out_words = words; a.dbg_err = &g_dbg_err;
  std::vector<const uint64_t *> ip(items);
  std::vector<uint64_t *> op(items);
  for (uint32_t i = 0; i < items; i++) ip[i] = in + i * a.in_bs, op[i] = out + i * a.out_bs;
  a.in_ptrs = ip.data(); a.out_ptrs = op.data();
  a.gen_r[0] = r1; a.gen_r[1] = r2; a.gen_r[2] = r3;
  const unsigned gx = (lanes + 3) / 4;
  auto grid = [&](int nt, auto body) {
    for (unsigned y = 0; y < items; y++)
      for (unsigned x = 0; x < gx; x++) {
        blockIdx.x = x; blockIdx.y = y; blockIdx.z = 0;
        memset(sm, 0xA5, sizeof(sm));
        std::barrier<> bar(nt);
        g_bar = &bar;
        std::vector<std::thread> th;
        for (int t = 0; t < nt; t++) th.emplace_back([&body, t] { threadIdx.x = t; body(); });
        for (auto &t : th) t.join();
      }
  };
  if (!fixed) {
    if (inv) grid(GL_GEN_NT, [&a] { gl_generic_kernel<true>(a); });
    else grid(GL_GEN_NT, [&a] { gl_generic_kernel<false>(a); });
    return 0;
  }
#define SHAPE_F(R1, R2, R3, NT)                                                     \
  if (r1 == R1 && r2 == R2 && r3 == R3) {                                           \
    if (inv) grid(NT, [&a] { gl_pass3_kernel<R1, R2, R3, 4, NT, true, 1>(a); });     \
    else grid(NT, [&a] { gl_pass3_kernel<R1, R2, R3, 4, NT, false, 1>(a); });        \
    return 0;                                                                       \
  }
  SHAPES
  return -1;
}
"""


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    text = HARNESS.replace("  SHAPES\n", "".join("  SHAPE_F(%d, %d, %d, %d)\n" % s for s in shapes()))
    (d / "f.cpp").write_text(text)
    subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-shared", "-pthread", "-DGL_DEVICE_CHECKS",
                    "-I" + CSRC, "-I" + os.path.join(ROOT, "tests"), str(d / "f.cpp"), "-o", str(d / "f.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "f.so"))
    vp, i64, u32, u64 = ctypes.c_void_p, ctypes.c_int64, ctypes.c_uint32, ctypes.c_uint64
    lib.emu_fixed.argtypes = ([ctypes.c_int] * 5 + [vp, vp, u64, i64, i64, u32, u32] + [vp] * 5
                              + [i64, u32, u32, vp, vp, u64, u64, vp, u32])
    lib.emu_check_flags.restype = u32
    return lib


def test_both_directions_list_the_same_shapes():
    fwd, inv = (re.findall(r"ENTRY3M\(([\d, ]+),", open(os.path.join(CSRC, "gl_kern_small_%s.cu" % d)).read())
                for d in ("fwd", "inv"))
    assert fwd == inv and len(fwd) == len(shapes())


@pytest.mark.parametrize("shape", shapes(), ids=lambda s: "x".join(map(str, s[:3])))
@pytest.mark.parametrize("inv", [False, True])
def test_fixed_equals_run_time(emu, shape, inv):
    r, m = shape[:3], shape[0] * shape[1] * shape[2]
    lanes, C, items, n2 = 6, 2, 2, 3  # a full tile and half of one
    n = m * n2
    w = root(n, inv) if (P - 1) % n == 0 else root(m, inv)
    lo, hi = table(w, min(n, 4096), n if inv else 1), table(pow(w, 4096, P), (n + 4095) // 4096)
    full = np.stack([table(pow(w, k, P), lanes // C) for k in range(m)])
    one = table(root(m, inv), m)
    scaled = table(root(m, inv), m, 12345)
    ilo, ihi = table(7, 4096), table(pow(7, 4096, P), (n + 4095) // 4096)
    x = rand_field(m * lanes * items, seed=m + inv)
    x[:8] = 2**64 - 1
    mul = rand_field(m * lanes * items, seed=m + 7)
    rows, cols = (m, 1), (1, lanes)
    forms = [  # (strides, flags, first-round table, limit)
        (rows, 0, one, NOLIM), (rows, SCALE | MUL, scaled, NOLIM), (rows, PTR | MUL | MONT, one, NOLIM),
        (cols, LOAD_LF | STORE_LF | SCALE, scaled, NOLIM), (cols, LOAD_LF | STORE_LF | LOAD_CG | PTR, one, NOLIM),
        (cols, LOAD_LF | STORE_LF | PASS_TW, one, NOLIM), (cols, LOAD_LF | STORE_LF | PASS_TW | TW_TABLE, one, NOLIM),
        (cols, LOAD_LF | STORE_LF | PASS_TW | IN_TW, one, m // 2 + 1), (cols, STORE_LF, one, m - 1),
    ]
    for (ls, is_), flags, tw_m, limit in forms:
        got = []
        for fixed in (0, 1):
            out = np.zeros_like(x)
            assert emu.emu_fixed(*r, int(inv), fixed, x.ctypes.data, out.ctypes.data, x.size, ls, is_, lanes, flags,
                                 tw_m.ctypes.data, one.ctypes.data, lo.ctypes.data, hi.ctypes.data, full.ctypes.data,
                                 lanes // C, C, limit, ilo.ctypes.data, ihi.ctypes.data, n2,
                                 pow(n, P - 2, P) * 2**64 % P if inv else 0, mul.ctypes.data, items) == 0
            assert emu.emu_check_flags() == 0
            got.append(out)
        assert np.array_equal(got[0], got[1]), (flags, limit)
        assert got[0].any()
