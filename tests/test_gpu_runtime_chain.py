"""Runtime-chain kernels (lengths without a compiled instance): every tile form
at the sizes where it can go wrong, against the long-double oracle with the
suite's bounds (5e-7 log2 n FP32, 2e-15 log2 n FP64)."""
from __future__ import annotations

import numpy as np
import pytest

import mofft_b200 as m
import oracle
from tests.conftest import cuda_available, fp32_tol, fp64_tol, rel_l2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

CTYPE = {32: np.complex64, 64: np.complex128}

# (length, explicit chain or None, batch).  Staged tiles (one stage, short
# runs), direct rows of every register class, the thread limits, uneven radix
# orders, column passes whose last tile is partial, three passes.
CASES = [
    (14, None, 1), (21, None, 600), (28, [2, 14], 257), (39, [13, 3], 33), (63, None, 4),
    (77, None, 1001), (98, [7, 2, 7], 5), (108, None, 149), (143, None, 7), (210, None, 19),
    (343, None, 3), (450, [2, 15, 3, 5], 9), (1001, None, 2), (1536, [2, 16, 6, 8], 3),
    (2197, None, 5), (2744, [14, 14, 14], 2), (4095, None, 3), (5005, None, 2), (6561, None, 2),
    (9009, None, 1), (12005, None, 1),
    (4096, [2] * 12, 2),              # more butterflies than a CTA has threads
    # several butterflies per thread: uneven radices, small ones, the limits
    (35, None, 300), (243, None, 7), (500, None, 5), (2500, [10, 10, 5, 5], 3), (3125, None, 2),
    (4000, None, 3), (7007, None, 1), (12740, None, 2), (390625, None, 1),
    (28561, None, 3), (50625, None, 2), (30030, None, 1), (117649, None, 1), (531441, None, 1),
]


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n,chain,batch", CASES)
def test_runtime_chain(n, chain, batch, bits):
    import torch
    dist = n + 3
    buf = oracle.uniform(batch * dist, seed=n, dtype=CTYPE[bits])
    lines = buf.reshape(batch, dist)[:, :n].astype(np.complex128)
    x = torch.from_numpy(buf).cuda()
    tol = fp32_tol(n) if bits == 32 else fp64_tol(n)
    for direction in (m.FORWARD, m.BACKWARD):
        ref = oracle.fft_ld(lines, direction)
        for placement in (m.OUT_OF_PLACE, m.IN_PLACE):
            y = x.clone() if placement == m.IN_PLACE else torch.zeros_like(x)
            with m.Plan.create(n, direction, placement, bits=bits, batch=batch, distance=dist,
                               radices=chain) as plan:
                torch.cuda.synchronize()
                plan.execute(y if placement == m.IN_PLACE else x, y)
            out = y.cpu().numpy().reshape(batch, dist)
            assert rel_l2(out[:, :n], ref) <= tol, (direction, placement)
            gaps = buf.reshape(batch, dist)[:, n:] if placement == m.IN_PLACE else 0
            assert np.all(out[:, n:] == gaps)          # nothing outside the lines


def test_runtime_chain_dense_many_tiles():
    """Dense batches with many full tiles and a partial last one."""
    import torch
    for bits in (32, 64):
        for n, batch in ((20, 5000), (35, 4003), (100, 2001), (1000, 601), (3375, 301)):
            x = oracle.uniform(n * batch, seed=batch, dtype=CTYPE[bits]).reshape(batch, n)
            d = torch.from_numpy(x).cuda()
            y = torch.empty_like(d)
            with m.Plan.create(n, m.FORWARD, bits=bits, batch=batch) as plan:
                plan.execute(d, y)
            ref = oracle.fft_ld(x.astype(np.complex128), m.FORWARD)
            got = y.cpu().numpy()
            tol = fp32_tol(n) if bits == 32 else fp64_tol(n)
            per = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
            assert per.max() <= tol, (bits, n, int(np.argmax(per)))


@pytest.mark.parametrize("n,bits,error", [(343, 32, 1.0622e-7), (896, 32, 1.1022e-7),
                                          (3328, 32, 1.2079e-7), (343, 64, 1.9368e-16),
                                          (3328, 64, 2.1769e-16)])
def test_stage_twiddles_carry_no_extra_rounding(n, bits, error):
    """Relative L2 error against the long-double oracle with every stage twiddle
    looked up (`error`, over 2^17 points of uniform input; the spread between
    inputs is below 0.5 %).  Twiddles formed as products of two others have 2.1
    to 5.2 % more at these lengths."""
    import torch
    batch = (1 << 17) // n
    x = oracle.uniform(batch * n, seed=n + bits, dtype=CTYPE[bits]).reshape(batch, n)
    d = torch.from_numpy(x).cuda()
    y = torch.empty_like(d)
    with m.Plan.create(n, m.FORWARD, bits=bits, batch=batch) as plan:
        torch.cuda.synchronize()
        plan.execute(d, y)
    ref = oracle.fft_ld(x.astype(np.complex128), m.FORWARD)
    assert rel_l2(y.cpu().numpy(), ref) <= 1.015 * error


@pytest.mark.parametrize("n,other,bits,limit", [(6825, 6930, 64, 5.85), (12870, 3375, 32, 14.1)])
def test_ping_pong_kernel_keeps_its_arguments(n, other, bits, limit):
    """Lengths whose chains ask for more threads than a runtime tile has run the
    ping-pong kernel: their time per point over that of a length with a runtime
    tile, both bound by issue.  322 / 62.4 us per 2^22 FP64 points and 472 / 37.2
    per 2^23 FP32 points where this was written; 414 and 577 us with the
    ping-pong kernel's arguments copied to local memory, the limit half-way."""
    import torch
    points = 1 << (22 if bits == 64 else 23)
    stream = torch.cuda.Stream()

    def per_point(length):
        batch = points // length
        x = torch.zeros((batch, length), device="cuda",
                        dtype=torch.complex64 if bits == 32 else torch.complex128)
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        took = []
        with m.Plan.create(length, bits=bits, batch=batch) as plan, torch.cuda.stream(stream):
            plan.set_stream(stream.cuda_stream)
            for _ in range(12):
                start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                start.record()
                for _ in range(8):
                    plan.execute(x, y)
                end.record()
                end.synchronize()
                took.append(start.elapsed_time(end) / (length * batch))
        return min(took)
    per_point(other)                      # clocks up
    ratio = per_point(n) / per_point(other)
    assert ratio < limit, ratio
