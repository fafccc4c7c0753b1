"""Two-line column kernels: both sides of a split, aligned and odd starts, gaps
between the lines, against the long-double oracle with the suite's FP32 bound."""
from __future__ import annotations

import numpy as np
import pytest

import mofft_b200 as m
import oracle
from tests.conftest import cuda_available, fp32_tol, rel_l2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

TWIN = ["cols_float_320_t32_c16_tw", "cols_float_384_t32_c16_tw", "cols_float_512_t32_c16_tw"]


@pytest.mark.parametrize("name", TWIN)
@pytest.mark.parametrize("gap,start", [(0, 0), (0, 1), (3, 0), (2, 1)])
def test_twin_columns(name, gap, start):
    import torch
    kernels = {k["name"]: k for k in m.kernels()}
    for pair in ([name, name], [name, "cols_float_64_t4_c32_p"],
                 ["cols_float_64_t4_c32_p", name]):
        ks = [kernels[k] for k in pair]
        n, batch = ks[0]["length"] * ks[1]["length"], 2
        dist = n + gap
        buf = oracle.uniform(start + batch * dist, seed=n, dtype=np.complex64)
        lines = buf[start:].reshape(batch, dist)[:, :n].astype(np.complex128)
        x = torch.from_numpy(buf).cuda()
        for direction in (m.FORWARD, m.BACKWARD):
            ref = oracle.fft_ld(lines, direction)
            for placement in (m.OUT_OF_PLACE, m.IN_PLACE):
                y = x.clone() if placement == m.IN_PLACE else torch.zeros_like(x)
                src = y if placement == m.IN_PLACE else x
                with m.Plan.create(n, direction, placement, batch=batch, distance=dist,
                                   kernels=[k["index"] for k in ks]) as plan:
                    torch.cuda.synchronize()
                    plan.execute(src[start:], y[start:])
                out = y.cpu().numpy()[start:].reshape(batch, dist)
                assert rel_l2(out[:, :n], ref) <= fp32_tol(n), (pair, direction, placement)
                gaps = buf[start:].reshape(batch, dist)[:, n:] if placement == m.IN_PLACE else 0
                assert np.all(out[:, n:] == gaps)
