"""Batches in which polynomials share memory: found on the host (CPU), and
transformed one after another in the order the header states (GPU)."""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

from conftest import ROOT, from_dev, rand_field, to_dev

HARNESS = r"""
#include "gl_batch_plan.h"
extern "C" int shares(const gl_poly *p, uint64_t n) { return gl_batch_shares_memory(p, n); }
extern "C" void order(const gl_poly *p, uint64_t n, const uint8_t *plain, uint64_t *out) {
  std::vector<bool> f(plain, plain + n);
  const auto o = gl_batch_order(p, n, f);
  std::copy(o.begin(), o.end(), out);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("batch_plan")
    (d / "b.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "goldilocks_gb300", "csrc"), str(d / "b.cpp"), "-o", str(d / "b.so")],
                   check=True)
    return ctypes.CDLL(str(d / "b.so"))


def polys(spans):
    from goldilocks_gb300 import _lib as L
    arr = (L.Poly * len(spans))()
    for p, (at, n, d) in zip(arr, spans):
        p.data, p.len, p.dir = 4096 + 8 * at, n, d
    return arr


def test_sharing_is_found(plan):
    rng = random.Random(1)
    seen = set()
    for _ in range(2000):
        spans = [(rng.randrange(64), rng.choice([1, 2, 3, 4, 8]), 0) for _ in range(rng.randrange(1, 6))]
        if rng.random() < 0.3:
            spans.sort()
        words = [{at + i for i in range(n)} if n > 1 else set() for at, n, _ in spans]
        want = sum(map(len, words)) != len(set().union(*words))
        arr = polys(spans)
        assert bool(plan.shares(ctypes.byref(arr), ctypes.c_uint64(len(spans)))) == want, spans
        seen.add(want)
    assert seen == {True, False}


def test_sharing_is_found_in_any_order_and_spread(plan):
    rng = random.Random(2)
    seen = {True: 0, False: 0}
    for _ in range(600):
        reach = 1 << rng.randrange(6, 40)
        spans = [(rng.randrange(reach), rng.randrange(1, 2 + reach // rng.randrange(8, 4000)), 0)
                 for _ in range(rng.randrange(2, 60))]
        ends = sorted((at, at + n) for at, n, _ in spans if n > 1)
        want = any(b[0] < a[1] for a, b in zip(ends, ends[1:]))
        arr = polys(spans)
        assert bool(plan.shares(ctypes.byref(arr), ctypes.c_uint64(len(spans)))) == want, spans
        seen[want] += 1
    assert min(seen.values()) > 50


def test_order(plan):
    spans = [(0, 16, 1), (0, 8, 0), (0, 64, 0), (0, 16, 0), (0, 8, 1), (0, 32, 1), (0, 8, 0), (0, 16, 0)]
    plain = np.array([0, 0, 1, 0, 0, 1, 0, 0], dtype=np.uint8)
    out = np.zeros(8, dtype=np.uint64)
    arr = polys(spans)
    plan.order(ctypes.byref(arr), ctypes.c_uint64(8), plain.ctypes.data_as(ctypes.c_void_p),
               out.ctypes.data_as(ctypes.c_void_p))
    assert out.tolist() == [2, 5, 1, 6, 4, 3, 7, 0]


# (offset, length, direction) over one pool: a buffer in both directions, nested
# and half overlapping lengths of one and two passes, equal entries, a Rader length
# and one entry that shares nothing.
CASES = {
    "both directions": [(0, 1 << 14, 1), (0, 1 << 14, 0)],
    "equal entries": [(0, 4096, 0)] * 3 + [(8192, 512, 0)] * 2,
    "nested": [(0, 1 << 16, 0), (0, 1 << 12, 0), (1 << 15, 1 << 15, 1), (100, 240, 0), (1 << 17, 1 << 12, 0)],
    "half over": [(0, 1 << 13, 0), (1 << 12, 1 << 13, 1), (1 << 13, 1 << 12, 0), (5, 257 * 16, 0)],
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("mode", ["AUTO", "BUCKETS", "PERSISTENT", "PER_CALL"])
def test_one_after_another(gl, cuda, name, mode):
    from goldilocks_gb300 import batch
    spans = CASES[name]
    x = rand_field(1 << 18, seed=7)
    order = range(len(spans))
    if mode != "PER_CALL":
        order = sorted(order, key=lambda i: (spans[i][1] % 257 != 0, *(spans[i][1:] if spans[i][1] % 257 else ())))
    want = to_dev(cuda, x)
    for i in order:
        at, n, d = spans[i]
        (gl.intt if d else gl.ntt)(want[at:at + n])
    got = to_dev(cuda, x)
    batch.run_packed(got, *(np.array(v) for v in zip(*spans)), mode=getattr(batch, mode))
    assert np.array_equal(from_dev(got), from_dev(want))
