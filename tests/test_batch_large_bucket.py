"""More polynomials of one length than a launch's grid.y holds."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HARNESS = r"""
#include "gl_batch_plan.h"
extern "C" uint64_t runs(const uint64_t *len, const int *dir, uint64_t n, uint64_t most, uint64_t *out) {
  std::vector<std::pair<uint64_t, int>> sig;
  for (uint64_t i = 0; i < n; i++) sig.push_back({len[i], dir[i]});
  const auto r = gl_bucket_runs(sig, most);
  for (size_t i = 0; i < r.size(); i++) out[2 * i] = r[i].first, out[2 * i + 1] = r[i].second;
  return r.size();
}
"""


@pytest.mark.parametrize("counts", [[1], [7], [8], [15, 1, 14], [3, 7, 8, 21], []])
def test_runs(tmp_path, counts):
    (tmp_path / "r.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "goldilocks_gb300", "csrc"), str(tmp_path / "r.cpp"),
                    "-o", str(tmp_path / "r.so")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "r.so"))
    lib.runs.restype = ctypes.c_uint64
    lens = np.repeat(np.arange(len(counts), dtype=np.uint64) // 2, counts)  # two directions of a length
    dirs = np.repeat(np.arange(len(counts), dtype=np.int32) % 2, counts)
    out = np.zeros(2 * (len(lens) + 1), dtype=np.uint64)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    k = lib.runs(p(lens), p(dirs), ctypes.c_uint64(len(lens)), ctypes.c_uint64(7), p(out))
    got = out[:2 * k].reshape(-1, 2).tolist()
    want, at = [], 0
    for c in counts:
        want += [[at + i, at + min(i + 7, c)] for i in range(0, c, 7)]
        at += c
    assert got == want


@pytest.mark.gpu
@pytest.mark.parametrize("n,count", [(4, 65535), (4, 65537), (64, 131073), (4096, 65537)])
def test_words(gl, cuda, n, count):
    from goldilocks_gb300 import batch
    gen = cuda.Generator(device="cuda").manual_seed(count)
    got = cuda.randint(0, 2**62, (n * (count + 3),), dtype=cuda.int64, device="cuda", generator=gen)
    want = got.clone()
    gl.strategy(n).ntt(want[:n * count])
    gl.strategy(n).intt(want[n * count:])
    batch.run_packed(got, n * np.arange(count + 3), np.full(count + 3, n), np.arange(count + 3) >= count,
                     mode=batch.BUCKETS)
    assert cuda.equal(got, want)
