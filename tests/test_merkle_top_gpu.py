"""GPU: trees whose layers lie at the edges of the kernels that take one warp
per block (at most 2048 blocks) and the top of a tree (at most 16 blocks), on
inputs on and off the 16-byte boundary, and trees one after another into the
same buffer, against the oracle."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [33, 40, 159, 160, 161, 163, 166, 160 * 15 + 5, 160 * 16, 160 * 16 + 1, 160 * 17, 800 * 16, 800 * 16 + 9,
           160 * 2048, 160 * 2048 + 1, 800 * 2048 - 1, 800 * 2048, 800 * 2048 + 1, 800 * 2049,
           4000 * 128 + 7]


@pytest.mark.parametrize("length", LENGTHS)
def test_tree_lengths(gl, oracle, cuda, length):
    from goldilocks_gb300 import k12
    data = np.random.default_rng(length).integers(0, 256, size=length, dtype=np.uint8)
    want = oracle.merkle_tree(data.tobytes())
    for shift in (0, 1, 8):
        buf = cuda.zeros(length + shift, dtype=cuda.uint8, device="cuda")
        buf[shift:] = cuda.from_numpy(data.copy()).cuda()
        got = [x.cpu().numpy().tobytes() for x in k12.merkle_tree(buf[shift:])]
        assert got == want, shift


def test_trees_back_to_back_in_one_buffer(gl, oracle, cuda):
    """Each call rewrites the layers the one before it read: no layer may come
    from the earlier tree (output off the 32-byte boundary as well)."""
    from goldilocks_gb300 import _lib as L
    lib, length = L.load(), 800 * 700 + 3
    total = lib.gl_merkle_tree_bytes(length)
    data = [np.random.default_rng(i).integers(0, 256, size=length, dtype=np.uint8) for i in range(4)]
    dev = [cuda.from_numpy(d).cuda() for d in data]
    for shift in (0, 8):
        out = cuda.zeros(total + shift, dtype=cuda.uint8, device="cuda")[shift:]
        got = []
        for d in dev * 3:
            assert lib.gl_merkle_tree(d.data_ptr(), length, out.data_ptr(), total, L.GL_MEM_DEVICE,
                                      ctypes.c_void_p(cuda.cuda.current_stream().cuda_stream)) == 0
            got.append(out.clone())
        for i, g in enumerate(got):
            assert g.cpu().numpy().tobytes() == b"".join(oracle.merkle_tree(data[i % 4].tobytes())), (shift, i)
