"""GPU: single-pass calls over more than 2^32 - 1 transforms or columns (64 GiB),
whose lane numbers do not fit 32 bits."""
import pytest

from conftest import P

pytestmark = pytest.mark.gpu

MORE = 77  # beyond 2^32


@pytest.fixture
def words(cuda):
    n = 2 * ((1 << 32) + MORE)
    cuda.cuda.empty_cache()
    if cuda.cuda.mem_get_info()[0] < 8 * n + (8 << 30):
        pytest.skip("needs 72 GiB of device memory")
    x = cuda.empty(n, dtype=cuda.int64, device="cuda")
    yield x
    del x
    cuda.cuda.empty_cache()


def spots():
    """First lanes, lanes around the edges of a launch and the last ones."""
    return [0, 1, 63, (1 << 32) - 257, (1 << 32) - 256, (1 << 32) - 1, 1 << 32, (1 << 32) + 1, (1 << 32) + MORE - 1]


def check(first, second, a, b):
    want = ((a + b) % P, (a - b) % P)
    assert (first % 2**64, second % 2**64) == want, (a, b)


def test_transforms(gl, words):
    x = words
    x[0::2], x[1::2] = 5, 3
    for i, l in enumerate(spots()):
        x[2 * l], x[2 * l + 1] = 1000 + i, 17 + 3 * i
    gl.strategy(2).ntt(x)
    for i, l in enumerate(spots()):
        check(int(x[2 * l]), int(x[2 * l + 1]), 1000 + i, 17 + 3 * i)
    assert int((x[0::2] != 8).sum()) == int((x[1::2] != 2).sum()) == len(spots())


def test_columns(gl, words):
    from goldilocks_gb300 import _lib as L
    x = words
    c = x.numel() // 2
    x[:c], x[c:] = 5, 3
    for i, l in enumerate(spots()):
        x[l], x[c + l] = 1000 + i, 17 + 3 * i
    assert L.load().gl_ntt_columns(x.data_ptr(), 2, c, L.GL_FORWARD, L.GL_MEM_DEVICE, None) == L.GL_OK
    for i, l in enumerate(spots()):
        check(int(x[l]), int(x[c + l]), 1000 + i, 17 + 3 * i)
    assert int((x[:c] != 8).sum()) == int((x[c:] != 2).sum()) == len(spots())
