"""Two-line one-pass kernels: odd starts, gaps between the lines and unpaired last
lines, and the errors of short lines, against the long-double oracle."""
from __future__ import annotations

import numpy as np
import pytest

import mofft_b200 as m
import oracle
from tests.conftest import cuda_available, fp32_tol, rel_l2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

CTYPE = {32: np.complex64, 64: np.complex128}


def twin_rows():
    return [k for k in m.kernels() if k["name"].startswith("rows_float") and "_tw" in k["name"]]


@pytest.mark.parametrize("batch,gap,start", [(1, 0, 1), (33, 0, 1), (32, 3, 0), (65, 1, 3)])
def test_twin_rows(batch, gap, start):
    import torch
    assert len(twin_rows()) >= 10
    for k in twin_rows():
        n, dist = k["length"], k["length"] + gap
        buf = oracle.uniform(start + batch * dist, seed=n, dtype=np.complex64)
        lines = buf[start:].reshape(batch, dist)[:, :n].astype(np.complex128)
        x = torch.from_numpy(buf).cuda()
        for direction in (m.FORWARD, m.BACKWARD):
            ref = oracle.fft_ld(lines, direction)
            for placement in (m.OUT_OF_PLACE, m.IN_PLACE):
                y = x.clone() if placement == m.IN_PLACE else torch.zeros_like(x)
                src = y if placement == m.IN_PLACE else x
                with m.Plan.create(n, direction, placement, batch=batch, distance=dist,
                                   kernels=[k["index"]]) as plan:
                    torch.cuda.synchronize()
                    plan.execute(src[start:], y[start:])
                out = y.cpu().numpy()
                got = out[start:].reshape(batch, dist)
                per = (np.linalg.norm(got[:, :n] - ref, axis=1) / np.linalg.norm(ref, axis=1))
                assert per.max() <= fp32_tol(n), (k["name"], direction, placement)
                kept = buf if placement == m.IN_PLACE else np.zeros_like(buf)
                assert np.array_equal(out[:start], kept[:start])
                assert np.array_equal(got[:, n:], kept[start:].reshape(batch, dist)[:, n:])


@pytest.mark.parametrize("n,bits,error", [(64, 32, 8.053e-8), (128, 32, 8.754e-8),
                                          (256, 32, 9.524e-8), (128, 64, 1.616e-16)])
def test_short_lines_carry_no_extra_rounding(n, bits, error):
    """Relative L2 error with every stage twiddle looked up (`error`, over 2^17
    points of uniform input; the spread between inputs is below 0.5 %).
    Twiddles formed as products have 4.5 to 5.4 % more at these lengths."""
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
