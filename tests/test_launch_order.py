"""CPU: a pass kernel marked late lets the next kernel of its stream start only
after its own wait, and every other one before it, so that waiting kernels do not
fill the SMs in a chain."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "goldilocks_gb300", "csrc")


@pytest.mark.parametrize("name", ["gl_pass3.cuh", "gl_generic.cuh"])
def test_order(name):
    src = open(os.path.join(CSRC, name)).read()
    calls = [m.group(0) for m in re.finditer(r"(if \([^;]*\) )?gl_pdl_\w+\(\);", src)]
    assert calls == ["if (!(a.flags & GL_PF_LATE)) gl_pdl_launch_dependents();", "gl_pdl_wait();",
                     "if (a.flags & GL_PF_LATE) gl_pdl_launch_dependents();"]
