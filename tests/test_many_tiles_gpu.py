"""GPU: passes compiled in two forms (few tiles, many tiles) give the same
words: 512 x m transforms ten at a time (1280 row tiles, more than eight per SM)
against one at a time (128 tiles), and one of them against the oracle."""
import numpy as np
import pytest

from conftest import rand_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [320, 340, 384, 408, 480, 544, 640, 680, 768, 1024, 1088, 1280, 1360, 1536, 1920, 2040, 2048, 2176, 2560, 2720, 3072, 3264])
@pytest.mark.parametrize("inv", [False, True])
def test_many_tiles_equal_few(oracle, m, inv):
    import torch

    import goldilocks_gb300 as gl
    n = 512 * m
    x = rand_field(10 * n, seed=m + inv)
    many = torch.from_numpy(x.view(np.int64).copy()).cuda()
    plan = gl.strategy(n)
    run = plan.intt if inv else plan.ntt
    run(many)
    got = many.cpu().numpy().view(np.uint64).reshape(10, n)
    for i in range(10):
        one = torch.from_numpy(x[i * n:(i + 1) * n].view(np.int64).copy()).cuda()
        run(one)
        assert np.array_equal(one.cpu().numpy().view(np.uint64), got[i]), i
    assert np.array_equal((oracle.intt if inv else oracle.ntt)(x[n:2 * n].copy()), got[1])
