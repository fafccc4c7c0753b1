"""Host-buffer executes: the first calls of a plan are staged, later small ones
run on mapped pinned memory; both against the oracle, at the limits of that
path (its call count, its span, gaps between transforms, one-pass only)."""
from __future__ import annotations

import numpy as np
import pytest

import mofft_b200 as m
import oracle
from tests.conftest import cuda_available, fp32_tol, fp64_tol, rel_l2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

CTYPE = {32: np.complex64, 64: np.complex128}


@pytest.mark.parametrize("n,batch,gap", [(16, 1, 0), (1000, 3, 5), (1024, 64, 0), (1024, 65, 0),
                                         (8192, 4, 0), (16384, 1, 0), (32768, 1, 0)])
@pytest.mark.parametrize("bits", [32, 64])
def test_repeated_host_executes(n, batch, gap, bits):
    dist = n + gap
    tol = fp32_tol(n) if bits == 32 else fp64_tol(n)
    for placement in (m.OUT_OF_PLACE, m.IN_PLACE):
        with m.Plan.create(n, m.BACKWARD, placement, bits=bits, batch=batch,
                           distance=dist) as plan:
            for call in (1, 31, 32, 33, 40):
                while getattr(plan, "calls", 0) < call:
                    plan.calls = getattr(plan, "calls", 0) + 1
                    buf = oracle.uniform(batch * dist, seed=plan.calls, dtype=CTYPE[bits])
                    out = buf.copy() if placement == m.IN_PLACE else np.zeros_like(buf)
                    plan.execute(out if placement == m.IN_PLACE else buf, out)
                lines = buf.reshape(batch, dist)[:, :n].astype(np.complex128)
                got = out.reshape(batch, dist)[:, :n]
                assert rel_l2(got, oracle.fft_ld(lines, m.BACKWARD)) <= tol, (placement, call)


@pytest.mark.parametrize("n,batch,gap", [(16, 3, 1), (1000, 3, 5), (256, 200, 7), (32768, 2, 3),
                                         (4096, 1000, 4)])
@pytest.mark.parametrize("bits", [32, 64])
def test_gaps_between_transforms_stay(n, batch, gap, bits):
    """A strided host execute writes its transforms and nothing between them,
    staged in one chunk or several (the last case) and on the mapped span."""
    dist = n + gap
    calls = (1, 2, 31, 32, 40) if batch * dist * bits // 4 <= 256 << 10 else (1, 2)
    for placement in (m.OUT_OF_PLACE, m.IN_PLACE):
        with m.Plan.create(n, m.FORWARD, placement, bits=bits, batch=batch,
                           distance=dist) as plan:
            for call in range(1, calls[-1] + 1):
                buf = oracle.uniform(batch * dist, seed=call, dtype=CTYPE[bits])
                out = buf.copy() if placement == m.IN_PLACE else np.full_like(buf, 3 - 5j)
                plan.execute(out if placement == m.IN_PLACE else buf, out)
                before = buf if placement == m.IN_PLACE else np.full_like(buf, 3 - 5j)
                got = out.reshape(batch, dist)
                assert np.array_equal(got[:, n:], before.reshape(batch, dist)[:, n:]), \
                    (placement, call)
                if call in calls:
                    ref = oracle.fft_ld(buf.reshape(batch, dist)[:, :n].astype(np.complex128), -1)
                    tol = fp32_tol(n) if bits == 32 else fp64_tol(n)
                    assert rel_l2(got[:, :n], ref) <= tol, (placement, call)


def test_mapped_memory_fits_the_plan():
    """64 small plans past their 32nd host call: 16 KiB of mapped memory each,
    which the driver cuts from chunks of 2 MiB."""
    def shared_kib():
        with open("/proc/self/status") as f:
            return next(int(line.split()[1]) for line in f if line.startswith("RssShmem"))

    x = oracle.uniform(1024, seed=1, dtype=np.complex64)
    out = np.empty_like(x)
    plans = [m.Plan.create(1024) for _ in range(64)]
    for plan in plans:
        for _ in range(31):
            plan.execute(x, out)
    before = shared_kib()
    for plan in plans:
        plan.execute(x, out)
    assert shared_kib() - before <= 2 * 2048
    assert rel_l2(out, oracle.fft_ld(x.astype(np.complex128), -1)) <= fp32_tol(1024)
