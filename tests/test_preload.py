"""CPU: every kernel outside the pass tables is in gl_preload_kernels' list, with
each instance that is launched."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "goldilocks_gb300", "csrc")
OWN = {"gl_tune.cu", "gl_debug.cu"}  # stated beside the list


def listed():
    text = "".join(open(f).read() for f in glob.glob(os.path.join(CSRC, "*.cu")))
    return set(re.findall(r"push_back\(\(const void \*\)(\w+(?:<\w+>)?)\)", text))


FILES = sorted(f for f in glob.glob(os.path.join(CSRC, "*.cu")) if os.path.basename(f) not in OWN)


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_kernels_are_listed(path):
    src = open(path).read()
    for name in re.findall(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", src):
        forms = set(re.findall(r"\b(%s<(?!<)\w+>)" % name, src)) or {name}
        assert forms <= listed(), forms - listed()


def test_lists_are_loaded():
    names = re.findall(r"^void (gl_\w+_kernels)\(std::vector<const void \*> &out\);",
                       open(os.path.join(CSRC, "gl_internal.h")).read(), re.M)
    body = open(os.path.join(CSRC, "gl_api.cu")).read().split("int gl_preload_kernels(void) {")[1].split("\n}\n")[0]
    assert len(names) >= 6
    for n in names:
        assert n + "(funcs);" in body, n
