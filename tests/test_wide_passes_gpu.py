"""GPU: passes of more lanes than the schedule's (large contiguous batches, host
memory, three-pass plans) give the words of the schedule's own kernels: counts
on both sides of the lines between them, against one transform at a time, host
memory against device memory, and the oracle."""
import numpy as np
import pytest

from conftest import rand_field

pytestmark = pytest.mark.gpu


def device(plan, x, inv):
    import torch
    t = torch.from_numpy(x.view(np.int64).copy()).cuda()
    (plan.intt if inv else plan.ntt)(t)
    return t.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("n,counts", [(1 << 13, (37, 38, 39, 460)), (1 << 14, (18, 20, 230)), (1 << 15, (9, 11)),
                                      (1 << 16, (57, 60)), (3 << 12, (30, 200)), (17 << 10, (40, 90)),
                                      (1 << 22, (1, 2)), (1 << 23, (1,))])
@pytest.mark.parametrize("inv", [False, True])
def test_contiguous_counts(oracle, n, counts, inv):
    import goldilocks_gb300 as gl
    plan = gl.strategy(n)
    x = rand_field(n * max(counts), seed=n % 1000 + inv)
    x[:64] = 2**64 - 1
    one = device(plan, x[:n], inv)
    last = device(plan, x[-n:], inv)
    assert np.array_equal(one, (oracle.intt if inv else oracle.ntt)(x[:n].copy()))
    for k in counts:
        got = device(plan, x[:n * k] if k < max(counts) else x, inv).reshape(k, n)
        assert np.array_equal(got[0], one)
        if k == max(counts):
            assert np.array_equal(got[-1], last)
            all_ = got.copy()
    for k in counts:
        assert np.array_equal(device(plan, x[:n * k], inv).reshape(k, n), all_[:k])


@pytest.mark.parametrize("n,count", [(1 << 17, 1), (1 << 18, 1), (1 << 19, 1), (1 << 20, 1), (1 << 21, 1), (1 << 13, 33),
                                     (1 << 16, 5), (3 << 18, 1), (17 << 15, 1), (1 << 22, 2)])
@pytest.mark.parametrize("inv", [False, True])
def test_host_memory_equals_device(n, count, inv):
    import torch
    import goldilocks_gb300 as gl
    plan = gl.strategy(n)
    x = rand_field(n * count, seed=n % 977 + inv)
    pinned = torch.from_numpy(x.view(np.int64).copy()).pin_memory()
    a = pinned.numpy().view(np.uint64)
    (plan.intt if inv else plan.ntt)(a)
    assert np.array_equal(a, device(plan, x, inv))


@pytest.mark.parametrize("n", [1 << 25, 255 << 17])
def test_three_passes(oracle, n):
    import torch
    import goldilocks_gb300 as gl
    plan = gl.strategy(n)
    x = rand_field(n, seed=25)
    got = device(plan, x, False)
    assert np.array_equal(got, oracle.ntt(x.copy()))
    assert np.array_equal(device(plan, got, True), x)
    a = torch.from_numpy(x.view(np.int64).copy()).pin_memory().numpy().view(np.uint64)
    plan.ntt(a)
    assert np.array_equal(a, got)


@pytest.mark.parametrize("n,cols", [(1 << 19, 24), (1 << 19, 32), (1 << 19, 30), (1 << 20, 32)])
@pytest.mark.parametrize("inv", [False, True])
def test_column_rows(n, cols, inv):
    import torch
    import goldilocks_gb300 as gl
    from goldilocks_gb300 import _lib
    x = rand_field(n * cols, seed=cols + inv).reshape(n, cols)
    t = torch.from_numpy(x.view(np.int64).copy()).cuda()
    assert _lib.load().gl_ntt_columns(t.data_ptr(), n, cols, _lib.GL_INVERSE if inv else _lib.GL_FORWARD,
                                      _lib.GL_MEM_DEVICE, torch.cuda.current_stream().cuda_stream) == _lib.GL_OK
    got = t.cpu().numpy().view(np.uint64)
    plan = gl.strategy(n)
    for c in range(0, cols, 3):
        assert np.array_equal(got[:, c], device(plan, np.ascontiguousarray(x[:, c]), inv)), c
