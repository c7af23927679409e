"""GPU: the profile records each kernel of a transform, a Rader step's too."""
import pytest

from conftest import rand_field, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,want", [
    (1 << 13, {"col 64 (8x8x1)": 1 << 13, "row 128 (16x8x1)": 1 << 13}),
    (257, {"rader 257": 257}),
    (257 * 16, {"rader 257": 257 * 16, "full 16 (16x1x1)": 257 * 16}),
])
def test_names(gl, cuda, n, want):
    from goldilocks_gb300 import _lib as L
    x = to_dev(cuda, rand_field(n, seed=n))
    gl.ntt(x)
    lib = L.load()
    lib.gl_profile_enable(1)
    try:
        gl.ntt(x)
        gl.ntt(x)
        ents = (L.ProfileEntry * 16)()
        n_ent = lib.gl_profile_read(ents, 16)
    finally:
        lib.gl_profile_enable(0)
    assert {e.name.decode(): (e.launches, e.elements) for e in ents[:n_ent]} == \
        {k: (2, 2 * v) for k, v in want.items()}
    assert all(e.total_ms > 0 for e in ents[:n_ent])
