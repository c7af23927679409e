"""GPU: a call starts while the kernel before it in its stream finishes
(programmatic dependent launch), and must still see everything ordered before
it: the kernel before it, of this library or not, copies and fills, events of
other streams, the legacy stream's order with blocking streams, and the
operations of a captured graph."""
import ctypes

import numpy as np
import pytest

from conftest import rand_field

pytestmark = pytest.mark.gpu

# One pass (5 and 1000003-ish counts share sectors between CTAs), two passes,
# run-time radices, a Rader length, a three-pass length.
SIZES = [(5, 1001), (1 << 10, 1), (1 << 10, 333), (1 << 12, 1), (1 << 16, 1), (15 << 10, 1), (257 * 16, 1), (1 << 20, 1)]
WAIT = 400_000  # cycles a producer is held up: longer than any launch


def to_dev(torch, x):
    return torch.from_numpy(x.view(np.int64).copy()).cuda()


@pytest.fixture
def setup(gl, cuda):
    def make(n, count, seed=1):
        x = rand_field(n * count, seed=seed)
        dev = to_dev(cuda, x)
        plan = gl.strategy(n)
        want = dev.clone()
        plan.ntt(want)
        cuda.cuda.synchronize()
        return plan, dev, want
    return make


@pytest.mark.parametrize("n,count", SIZES)
def test_chains_of_calls(setup, cuda, n, count):
    plan, x, want = setup(n, count)
    y = x.clone()
    for i in range(60):
        plan.ntt(y)
        if i % 7 == 0:
            assert cuda.equal(y, want), i
        plan.intt(y)
    assert cuda.equal(y, x)
    out = []
    for _ in range(20):  # the producer is a kernel of another library
        z = x ^ 1
        z ^= 1
        plan.ntt(z)
        out.append(z)
    assert all(cuda.equal(z, want) for z in out)


@pytest.mark.parametrize("n,count", SIZES)
def test_late_producers(setup, cuda, n, count):
    plan, x, want = setup(n, count)
    s1, s2 = cuda.cuda.Stream(), cuda.cuda.Stream()
    pinned = x.cpu().pin_memory()
    for _ in range(5):
        # an event of another stream between two calls
        y, other = cuda.zeros_like(x), x.clone()
        cuda.cuda.synchronize()
        with cuda.cuda.stream(s1):
            cuda.cuda._sleep(WAIT)
            y.copy_(x)
            e = s1.record_event()
        with cuda.cuda.stream(s2):
            plan.ntt(other)
            s2.wait_event(e)
            plan.ntt(y)
        s2.synchronize()
        assert cuda.equal(y, want) and cuda.equal(other, want)
        # a kernel, a fill and a copy right before the call
        with cuda.cuda.stream(s2):
            a, b, c = cuda.zeros_like(x), cuda.ones_like(x), cuda.zeros_like(x)
            cuda.cuda._sleep(WAIT)
            a.add_(x)
            plan.ntt(a)
            cuda.cuda._sleep(WAIT)
            b.zero_()
            plan.ntt(b)
            c.copy_(pinned, non_blocking=True)
            plan.ntt(c)
        s2.synchronize()
        assert cuda.equal(a, want) and not b.any() and cuda.equal(c, want)


@pytest.mark.parametrize("n,count", [(1 << 10, 333), (1 << 16, 1), (257 * 16, 1)])
def test_legacy_stream_waits_for_blocking_streams(setup, cuda, gl, n, count):
    from goldilocks_gb300 import _lib as L
    plan, x, want = setup(n, count)
    rt = ctypes.CDLL("libcudart.so.13")
    h = ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(h)) == 0  # a blocking stream
    s = cuda.cuda.ExternalStream(h.value)
    lib = L.load()
    for _ in range(10):
        y, other = cuda.zeros_like(x), x.clone()
        cuda.cuda.synchronize()
        assert lib.gl_plan_execute(plan._h, other.data_ptr(), x.numel(), 0, L.GL_MEM_DEVICE, None) == 0
        with cuda.cuda.stream(s):
            cuda.cuda._sleep(WAIT)
            y.copy_(x)
        assert lib.gl_plan_execute(plan._h, y.data_ptr(), x.numel(), 0, L.GL_MEM_DEVICE, None) == 0
        cuda.cuda.synchronize()
        assert cuda.equal(y, want) and cuda.equal(other, want)
    del s
    assert rt.cudaStreamDestroy(h) == 0


@pytest.mark.parametrize("n,count", SIZES)
def test_captured_calls(setup, cuda, n, count):
    plan, x, want = setup(n, count)
    y, z = x.clone(), cuda.zeros_like(x)
    ws = cuda.empty(max(1, 2 * plan.workspace_bytes(count) // 8), dtype=cuda.int64, device="cuda")
    from goldilocks_gb300 import _lib as L
    lib = L.load()

    def run(t, d, half):
        need = plan.workspace_bytes(count)
        assert lib.gl_plan_execute_ws(plan._h, t.data_ptr(), t.numel(), d, ws[half * (need // 8):].data_ptr(), need,
                                      cuda.cuda.current_stream().cuda_stream) == 0

    main, side = cuda.cuda.Stream(), cuda.cuda.Stream()
    g = cuda.cuda.CUDAGraph()
    cuda.cuda.synchronize()
    with cuda.cuda.graph(g, stream=main):
        y.copy_(x)
        run(y, 0, 0)
        e = main.record_event()
        with cuda.cuda.stream(side):  # forked, and joined before the next call
            side.wait_event(e)
            z.zero_()
            z.add_(x)
            run(z, 0, 1)
            j = side.record_event()
        run(y, 1, 0)
        main.wait_event(j)
        run(z, 1, 0)
        run(z, 0, 0)
    for _ in range(5):
        y.zero_()
        z.zero_()
        g.replay()
        cuda.cuda.synchronize()
        assert cuda.equal(y, x) and cuda.equal(z, want)


@pytest.mark.parametrize("n,count", [(1 << 10, 3), (1 << 16, 1), (1 << 12, 5)])
def test_factors_written_by_the_call_before(gl, cuda, n, count):
    b = to_dev(cuda, rand_field(n, seed=5))
    a = to_dev(cuda, rand_field(n * count, seed=6))
    hat = b.clone()
    gl.ntt(hat)
    want = a.clone()
    cuda.cuda.synchronize()
    gl.convolve(want, hat, size=n)
    cuda.cuda.synchronize()
    for _ in range(40):
        hat2, got = b.clone(), a.clone()
        gl.ntt(hat2)
        gl.convolve(got, hat2, size=n)
        assert cuda.equal(got, want)
