"""The codelets' lazy arithmetic (three unreduced limbs, gl_field.cuh): the
operations on the host against Python integers, and on the GPU transforms of
words at the edges of the limbs (all-ones words, words at and above p, single
set bits), where a carry, a borrow or a fold goes wrong if it can, through
every codelet radix."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import P, ROOT

EDGE = [0, 1, 2, 2**31, 2**32 - 1, 2**32, 2**32 + 1, 2**63, P - 1, P, P + 1, 2**64 - 2**32, 2**64 - 1,
        0xffffffff00000000, 0x00000000fffffffe, 0x8000000080000000]

HARNESS = r"""
#include "gl_codelets.cuh"
static gl_l3 in(const uint32_t *v) { return {v[0], v[1], v[2]}; }
static void put(gl_l3 r, uint32_t *o) { o[0] = r.x0; o[1] = r.x1; o[2] = r.x2; }
extern "C" {
void l_add(const uint32_t *a, const uint32_t *b, uint32_t *o) { put(gl_ladd(in(a), in(b)), o); }
void l_sub(const uint32_t *a, const uint32_t *b, uint32_t *o) { put(gl_lsub(in(a), in(b)), o); }
void l_norm(const uint32_t *a, uint32_t *o) { put(gl_lnorm(in(a)), o); }
void l_bias(const uint32_t *a, uint32_t *o) { put(gl_lbias<12345>(in(a)), o); }
void l_negb(const uint32_t *a, uint32_t *o) { put(gl_lnegb<12345>(in(a)), o); }
uint64_t l_fold(const uint32_t *a) { return gl_lfold(in(a)); }
int l_shl(int k, const uint32_t *a, uint32_t *o) {
  switch (k) {
%CASES%
  }
  return -1;
}
}
"""
SHIFTS = [3, 12, 24, 30, 32, 36, 48, 60, 63, 64, 72, 84, 93]


def value(v):
    x2 = int(v[2])
    return int(v[0]) + (int(v[1]) << 32) + ((x2 - 2**32 if x2 >> 31 else x2) << 64)


def limbs(x):
    return np.array([x & 0xffffffff, (x >> 32) & 0xffffffff, (x >> 64) & 0xffffffff], dtype=np.uint32)


def test_operations_on_the_host(tmp_path):
    cases = "\n".join("  case %d: put(gl_lshl<%d>(in(a)), o); return 0;" % (k, k) for k in SHIFTS)
    src, so = tmp_path / "l.cpp", tmp_path / "l.so"
    src.write_text(HARNESS.replace("%CASES%", cases))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "goldilocks_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.l_fold.restype = ctypes.c_uint64
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    out = np.zeros(3, dtype=np.uint32)
    rng = np.random.default_rng(5)
    words = EDGE + [int(v) for v in rng.integers(0, 2**64, 12, dtype=np.uint64)]
    vals = [w + (h << 64) for w in words for h in (-2**20, -2, -1, 0, 1, 3, 2**20)]
    for i, a in enumerate(vals):
        la = limbs(a)
        for b in vals[i % 11::11]:
            lb = limbs(b)
            lib.l_add(ptr(la), ptr(lb), ptr(out))
            assert value(out) == a + b
            lib.l_sub(ptr(la), ptr(lb), ptr(out))
            assert value(out) == a - b
        lib.l_norm(ptr(la), ptr(out))
        assert (value(out) - a) % P == 0 and abs(value(out) >> 64) <= 1
        lib.l_bias(ptr(la), ptr(out))
        assert value(out) == a + 12345 * P
        lib.l_negb(ptr(la), ptr(out))
        assert value(out) == 12345 * P - a
        if a >= 0:
            assert (lib.l_fold(ptr(la)) - a) % P == 0
        for k in SHIFTS:
            if abs(a) << (k % 32) < 2**95:  # the shifted value fits three limbs
                assert lib.l_shl(k, ptr(la), ptr(out)) == 0
                assert (value(out) - a * 2**k) % P == 0, (hex(a), k)


# Every codelet radix as a whole transform, then tiles of two and three rounds
# (compiled, Good-Thomas and run-time radices) and a Rader length.
LENGTHS = [2, 3, 4, 5, 6, 8, 10, 12, 15, 16, 17, 32, 60, 64, 68, 128, 255, 256, 272, 512, 680, 1536, 2048, 4096,
           5 << 12, 51 << 10, 65536, 85 << 10, 4080 << 4, 257 * 16]


@pytest.mark.gpu
@pytest.mark.parametrize("inv", [False, True])
@pytest.mark.parametrize("n", LENGTHS)
def test_edge_words_on_the_gpu(oracle, n, inv):
    import torch

    import goldilocks_gb300 as gl
    rng = np.random.default_rng(n)
    edge = np.array(EDGE, dtype=np.uint64)
    rows = [edge[rng.integers(0, len(edge), n)], np.full(n, 2**64 - 1, dtype=np.uint64),
            np.full(n, P - 1, dtype=np.uint64), edge[np.arange(n) % len(edge)]]
    x = np.concatenate(rows)
    dev = torch.from_numpy(x.view(np.int64).copy()).cuda()
    plan = gl.strategy(n)
    (plan.intt if inv else plan.ntt)(dev)
    got = dev.cpu().numpy().view(np.uint64).reshape(len(rows), n)
    for r, row in enumerate(rows):
        canon = np.where(row >= np.uint64(P), row - np.uint64(P), row)
        assert np.array_equal(got[r], (oracle.intt if inv else oracle.ntt)(canon)), r
