"""GPU: bucket batches of more buckets than graph branches, with lengths of
every kind (one transform per CTA, one to three passes, run-time radices, a
Rader step, length 1), replayed on other data, against single transforms."""
import numpy as np
import pytest

from conftest import rand_field

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 16, 256, 512, 1024, 2048, 4096, 60, 272, 8192, 1 << 14, 1 << 16, 15 << 9, 51 << 9, 257 * 4, 17 << 12]


@pytest.mark.parametrize("repeat", [1, 3])
def test_many_buckets(gl, cuda, repeat):
    from goldilocks_gb300 import batch
    rng = np.random.default_rng(repeat)
    lens = [n for n in LENGTHS for _ in range(repeat) for _ in (0, 1)]
    dirs = [d for _ in LENGTHS for _ in range(repeat) for d in (batch.FORWARD, batch.INVERSE)]
    order = rng.permutation(len(lens))
    lens, dirs = [lens[i] for i in order], [dirs[i] for i in order]
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    for seed in range(3):  # captured once, replayed with other pools
        x = rand_field(int(sum(lens)), seed=seed)
        pool = cuda.from_numpy(x.view(np.int64).copy()).cuda()
        want = pool.clone()
        for o, n, d in zip(offs, lens, dirs):
            (gl.ntt if d == batch.FORWARD else gl.intt)(want[o:o + n])
        batch.run_packed(pool, offs, lens, dirs, mode=batch.BUCKETS)
        assert cuda.equal(pool, want), seed
