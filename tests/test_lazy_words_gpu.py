"""GPU: the codelets' three-limb operations (gl_field.cuh, inline PTX), each
alone, at the edges of the limbs against Python integers.  The top limb is
compared modulo 2^32 where nothing bounds it, the value where the operation only
keeps it modulo p."""
import numpy as np
import pytest

from conftest import P, from_dev, to_dev
from test_lazy_words import EDGE, SHIFTS

pytestmark = pytest.mark.gpu

TOPS = [0, 1, 2, 3, 2**20, 2**31 - 1, 2**31, 2**32 - 2**20, 2**32 - 2, 2**32 - 1]


def signed(x):
    x %= 2**96
    return x - 2**96 if x >> 95 else x


@pytest.fixture(scope="module")
def operands():
    """Every edge word with every edge top limb, and uniform ones."""
    rng = np.random.default_rng(11)
    words = EDGE + [int(v) for v in rng.integers(0, 2**64, 40, dtype=np.uint64)]
    pairs = [(w, t << 32 | low) for w in words for t in TOPS + [int(v) for v in rng.integers(0, 2**32, 6)]
             for low in (0, 1, 2**31, 2**32 - 1, int(rng.integers(0, 2**32)))]
    a, b = (np.array(v, dtype=np.uint64) for v in zip(*pairs))
    return a, b


def run(gl, cuda, f, a, b):
    """The three limbs of the result as a signed integer."""
    lib, parts = gl._lib.load(), []
    da, db = to_dev(cuda, a), to_dev(cuda, b)
    for part in (0, 1):
        out = cuda.empty(a.size, dtype=cuda.int64, device="cuda")
        assert lib.gl_debug_field_op(gl._lib.GL_FOP_LAZY + 2 * f + part, da.data_ptr(), db.data_ptr(),
                                     out.data_ptr(), a.size, cuda.cuda.current_stream().cuda_stream) == gl._lib.GL_OK
        parts.append(from_dev(out).tolist())
    return [signed(lo + (hi << 64)) for lo, hi in zip(*parts)]


@pytest.mark.parametrize("f", range(8))
def test_operations(gl, cuda, operands, f):
    a, b = operands
    for x, y, got in zip(a.tolist(), b.tolist(), run(gl, cuda, f, a, b)):
        v, w = signed(x + ((y >> 32) << 64)), signed(y + ((x % 2**32) << 64))
        if f < 6:
            want = [v + w, v - w, x + y, x - y, v + 12345 * P, 12345 * P - v][f]
            assert got == signed(want), (hex(x), hex(y))
        elif f == 6:
            assert (got - v) % P == 0 and -1 <= got >> 64 <= 1, (hex(x), hex(y))
        elif v >= 0:
            assert 0 <= got < 2**64 and (got - v) % P == 0, (hex(x), hex(y))


@pytest.mark.parametrize("k", SHIFTS)
def test_shifts(gl, cuda, operands, k):
    a, b = operands
    seen = 0
    for x, y, got in zip(a.tolist(), b.tolist(), run(gl, cuda, 8 + k, a, b)):
        v = signed(x + ((y >> 32) << 64))
        if -2**95 <= v << (k % 32) < 2**95:  # the shifted limbs fit three
            assert (got - v * 2**k) % P == 0, (hex(x), hex(y))
            seen += 1
    assert seen > 400
