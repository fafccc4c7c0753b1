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
    workspace = 0

    def __init__(self):
        self._stream, self.log = None, []
        FakePlan.made.append(self)

    def set_stream(self, stream):
        self._stream = stream or None

    def execute(self, inp, out=None):
        self.log.append(("run", self._stream))

    def check_status(self):
        self.log.append(("wait", self._stream))

    def schedule(self):
        return {"workspace_bytes": FakePlan.workspace}


@pytest.fixture
def fakes(monkeypatch):
    """fft() on fake tensors, plans and streams; yields the stream's setter."""
    import torch
    FakePlan.made = []
    monkeypatch.setattr(FakePlan, "workspace", 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
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


@pytest.mark.parametrize("workspace", [0, 1 << 20])
def test_streams_share_no_workspace(fakes, monkeypatch, workspace):
    """A plan with a workspace runs on one stream only; one without runs on
    each call's stream.  A stream's second call finds its plan again."""
    import torch
    monkeypatch.setattr(FakePlan, "workspace", workspace)
    x = FakeTensor(65536, torch.complex64)
    for handle in (7, 9, 0, 7, 9, 0):
        fakes(handle)
        m.fft(x, inplace=True)
    ran = [[s for what, s in p.log if what == "run"] for p in FakePlan.made]
    assert ran == ([[7, 7], [9, 9], [1, 1]] if workspace else [[7, 9, 1, 7, 9, 1]])


@pytest.mark.parametrize("workspace", [0, 1 << 20])
def test_capture_makes_no_plan(fakes, monkeypatch, workspace):
    """A capture runs on a stream of its own and cannot allocate: it takes the
    plan that the shape's earlier call made, and leaves that call's stream its
    plan."""
    import torch
    monkeypatch.setattr(FakePlan, "workspace", workspace)
    x = FakeTensor(65536, torch.complex64)
    fakes(7)
    m.fft(x, inplace=True)
    fakes(9)
    with monkeypatch.context() as patch:
        patch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
        m.fft(x, inplace=True)
    fakes(7)
    m.fft(x, inplace=True)
    (plan,) = FakePlan.made
    assert [s for _, s in plan.log] == [7, 9, 7]


@pytest.mark.parametrize("workspace", [0, 1 << 20])
def test_threads_do_not_move_each_others_stream(fakes, monkeypatch, workspace):
    """Two threads on two streams, the second calling while the first one is
    inside its call: each transform runs on its own thread's stream."""
    import threading
    import torch
    monkeypatch.setattr(FakePlan, "workspace", workspace)
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
    real_set, turn = FakePlan.set_stream, threading.Barrier(2, timeout=0.2)

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


@pytest.mark.gpu
@needs_gpu
@pytest.mark.parametrize("n,batch,bits,inplace", [(1024, 64, 32, False), (65536, 8, 32, True),
                                                  (3375, 5, 64, False), (50625, 3, 64, True)])
def test_capture_after_a_warm_up(n, batch, bits, inplace):
    """The shape runs once on a side stream, then fft() is captured on the
    graph's own stream and replayed."""
    import torch
    dtype = np.complex64 if bits == 32 else np.complex128
    host = oracle.uniform(n * batch, seed=n, dtype=dtype).reshape(batch, n)
    src = torch.from_numpy(host).cuda()
    x = src.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        m.fft(x.clone(), inplace=inplace)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x.copy_(src)
        y = m.fft(x, inplace=inplace)
    for _ in range(2):
        y.zero_()
        graph.replay()
    torch.cuda.synchronize()
    ref = oracle.fft_ld(host.astype(np.complex128), -1)
    assert rel_l2(y.cpu().numpy(), ref) <= (fp32_tol(n) if bits == 32 else fp64_tol(n))
