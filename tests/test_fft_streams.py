"""The one-call fft and torch's streams: the order behind pending work, plans of
several streams and threads."""
from __future__ import annotations

import types

import numpy as np
import pytest

import mofft_b200 as m
import oracle
from tests.conftest import cuda_available, fp32_tol, fp64_tol, rel_l2

needs_gpu = pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")


class FakeTensor:
    """What fft() asks of a CUDA tensor."""
    is_cuda = True

    def __init__(self, n, dtype):
        self.shape, self.dtype, self.device = (n,), dtype, types.SimpleNamespace(index=0)

    def contiguous(self):
        return self

    def numel(self):
        return self.shape[0]

    def get_device(self):
        return 0


class FakePlan:
    """Records which stream it runs on, and the waits for it."""
    made: list = []

    def __init__(self):
        self._stream, self.log = None, []
        FakePlan.made.append(self)

    def set_stream(self, stream):
        self._stream = stream or None

    def execute(self, inp, out=None):
        self.log.append(("run", self._stream))

    def check_status(self):
        self.log.append(("wait", self._stream))


@pytest.fixture
def fakes(monkeypatch):
    """fft() on fake tensors, plans and streams; yields the stream's setter."""
    import torch
    FakePlan.made = []
    monkeypatch.setattr(m, "_PLAN_CACHE", {})
    monkeypatch.setattr(m.Plan, "create", lambda *a, **k: FakePlan())
    monkeypatch.setattr(torch, "empty_like", lambda x: x)
    waits = []

    def current(handle):
        stream = types.SimpleNamespace(cuda_stream=handle, synchronize=lambda: waits.append(handle))
        monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream)
        return waits
    return current


@pytest.mark.parametrize("bits", [32, 64])
def test_default_stream_keeps_its_order(fakes, bits):
    """On the default stream the transform is enqueued on that stream (its
    legacy handle is 1; handle 0 means the plan's own stream), then waited
    for."""
    import torch
    waits = fakes(0)
    m.fft(FakeTensor(1024, torch.complex64 if bits == 32 else torch.complex128))
    (plan,) = FakePlan.made
    assert plan.log[0] == ("run", 1)
    assert plan.log[1:] == ([("wait", 1)] if bits == 32 else []) and waits == [0] * (bits == 64)


@pytest.mark.gpu
@needs_gpu
@pytest.mark.parametrize("n,batch,bits", [(1024, 1, 32), (16384, 3, 32), (65536, 4, 32),
                                          (1000, 2, 64)])
@pytest.mark.parametrize("inplace", [False, True])
def test_default_stream_waits_for_the_input(n, batch, bits, inplace):
    """fft() right behind a slow producer of its input on the default stream."""
    import torch
    dtype = np.complex64 if bits == 32 else np.complex128
    host = oracle.uniform(n * batch, seed=n, dtype=dtype).reshape(batch, n)
    src = torch.from_numpy(host).cuda()
    x = torch.zeros_like(src)
    m.fft(x.clone(), inplace=inplace)         # the plan is made before the race
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)             # about 10 ms
    x.copy_(src)
    y = m.fft(x, inplace=inplace)
    ref = oracle.fft_ld(host.astype(np.complex128), -1)
    assert rel_l2(y.cpu().numpy(), ref) <= (fp32_tol(n) if bits == 32 else fp64_tol(n))
