"""CPU: a call takes its tensor's current stream, also from a torch that lacks the
private function for its handle."""
import importlib
import types

import pytest


@pytest.mark.parametrize("private", [True, False])
def test_handle(gl, monkeypatch, private):
    import torch
    ntt = importlib.import_module("goldilocks_gb300.ntt")

    class OnCuda(torch.Tensor):
        is_cuda = property(lambda self: True)

        def get_device(self):
            return 3

    if private:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 1000 + d, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
        monkeypatch.setattr(torch.cuda, "current_stream", lambda d: types.SimpleNamespace(cuda_stream=2000))
    x = torch.zeros(8, dtype=torch.int64).as_subclass(OnCuda)
    ptr, n, mem, stream = ntt._buffer(x)
    assert (ptr, n, mem, stream) == (x.data_ptr(), 8, gl._lib.GL_MEM_DEVICE, 1003 if private else 2000)
