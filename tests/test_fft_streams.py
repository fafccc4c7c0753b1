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


def test_streams_do_not_share_a_plan(fakes):
    """A plan may own a workspace: no plan runs on two streams, and a stream's
    second call finds its plan again."""
    import torch
    x = FakeTensor(65536, torch.complex64)
    for handle in (7, 9, 0, 7, 9, 0):
        fakes(handle)
        m.fft(x, inplace=True)
    ran = [[s for what, s in p.log if what == "run"] for p in FakePlan.made]
    assert ran == [[7, 7], [9, 9], [1, 1]]


def test_threads_do_not_move_each_others_stream(fakes, monkeypatch):
    """Two threads on two streams, the second calling while the first one is
    inside its call: each transform runs on its own thread's stream."""
    import threading
    import torch
    local = threading.local()
    monkeypatch.setattr(torch.cuda, "current_stream",
                        lambda device=None: types.SimpleNamespace(cuda_stream=local.handle))
    seen, lock = [], threading.Lock()
    real = FakePlan.execute

    def execute(self, inp, out=None):
        real(self, inp, out)
        with lock:
            seen.append((local.handle, self._stream))
    monkeypatch.setattr(FakePlan, "execute", execute)
    real_set, turn = FakePlan.set_stream, threading.Barrier(2, timeout=2)

    def set_stream(self, stream):
        real_set(self, stream)
        try:                                  # both threads have set theirs
            turn.wait()
        except threading.BrokenBarrierError:
            pass
    monkeypatch.setattr(FakePlan, "set_stream", set_stream)

    def work(handle):
        local.handle = handle
        for _ in range(50):
            m.fft(FakeTensor(65536, torch.complex64), inplace=True)
    threads = [threading.Thread(target=work, args=(h,)) for h in (7, 9)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(seen) == 100 and all(a == b for a, b in seen)


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


@pytest.mark.gpu
@needs_gpu
@pytest.mark.parametrize("n,batch,bits,inplace", [(65536, 64, 32, True), (50625, 40, 64, True),
                                                  (1 << 24, 1, 32, False),
                                                  (1 << 23, 1, 64, False)])
def test_streams_with_a_workspace(n, batch, bits, inplace):
    """Transforms of several passes with a workspace, on three streams at once
    (one of them the default one) and from two threads on one stream."""
    import threading
    import torch
    dtype = torch.complex64 if bits == 32 else torch.complex128
    real = torch.float32 if bits == 32 else torch.float64
    g = torch.Generator(device="cuda").manual_seed(n)

    def data():
        return torch.view_as_complex(torch.rand((batch, n, 2), generator=g, device="cuda",
                                                dtype=real) * 2 - 1)
    xs = [data() for _ in range(3)]
    refs = [m.fft(x) for x in xs]             # one at a time
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.default_stream()]

    def run(x, stream, out):
        with torch.cuda.stream(stream):
            out.extend(m.fft(x.clone() if inplace else x, inplace=inplace) for _ in range(4))
    outs = [[], [], []]
    for x, s in zip(xs, streams):
        s.wait_stream(torch.cuda.default_stream())
        run(x, s, outs[0])                    # make the plans
    torch.cuda.synchronize()
    for where in (streams, [streams[0]] * 2 + [streams[1]]):
        outs = [[], [], []]
        threads = [threading.Thread(target=run, args=a) for a in zip(xs, where, outs)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        for ref, got in zip(refs, outs):
            assert len(got) == 4
            for y in got:
                err = torch.linalg.vector_norm(y - ref) / torch.linalg.vector_norm(ref)
                # the same kernels on the same input; in place may run another schedule
                assert float(err) <= (fp32_tol(n) if bits == 32 else fp64_tol(n))
