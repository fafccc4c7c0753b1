"""Performance cases of the framework: what its users have it compute.

A case is one pass through the public Python entry points (which are thin
ctypes bindings of the C API): batched plans on device buffers, the one-call
``fft``, an in-place filtering step, host buffers, ragged batches and the
serving engine.  Lengths are those the library plans for: powers of two
2^4..2^24, 3*2^k and 5*2^k, and the other 13-smooth lengths (products of the
primes up to 13) that the reference publishes results for.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mofft_b200 as m
from mofft_b200 import workloads

FORWARD, BACKWARD = m.FORWARD, m.BACKWARD


def listed() -> list[dict]:
    return [
        # one short transform through the one-call interface: call latency
        {"name": "fft_1024_one", "kind": "fft", "n": 1024, "batch": 1, "bits": 32,
         "direction": FORWARD},
        # the reference's own calling convention: host arrays, one transform
        {"name": "host_1024_one", "kind": "host", "n": 1024, "batch": 1, "bits": 32,
         "direction": FORWARD},
        # a spectral method's pair of transforms on mid-size batches
        {"name": "roundtrip_f32_1024", "kind": "roundtrip", "n": 1024, "batch": 4096, "bits": 32,
         "direction": FORWARD},
        # the headline batch: 2^26 points, larger than L2
        {"name": "batch_f32_4096", "kind": "plan", "n": 4096, "batch": 16384, "bits": 32,
         "direction": FORWARD},
        # lengths that are no power of two: 15^3 in one pass, odd batch
        {"name": "smooth_f32_3375", "kind": "plan", "n": 3375, "batch": 4001, "bits": 32,
         "direction": FORWARD},
        # 15^4 in FP64, more than one pass, from spectrum back to samples
        {"name": "smooth_f64_50625", "kind": "plan", "n": 50625, "batch": 129, "bits": 64,
         "direction": BACKWARD},
        # 3*2^12: a frame length with a factor of three
        {"name": "batch_f32_12288", "kind": "plan", "n": 12288, "batch": 2730, "bits": 32,
         "direction": FORWARD},
        # FP64 inverse at the longest one-pass power of two
        {"name": "batch_f64_8192", "kind": "plan", "n": 8192, "batch": 2048, "bits": 64,
         "direction": BACKWARD},
        # an in-place propagation step: forward, all-pass filter, backward
        {"name": "filter_f32_65536", "kind": "filter", "n": 65536, "batch": 512, "bits": 32,
         "direction": FORWARD},
        # long transforms, three passes over memory
        {"name": "long_f32_1048576", "kind": "plan", "n": 1 << 20, "batch": 64, "bits": 32,
         "direction": FORWARD},
        # 512 transforms of mixed lengths, batch sizes and directions
        {"name": "ragged_512", "kind": "ragged", "count": 512, "spec": 7, "max_batch": 64},
        # a burst of requests to the serving engine, FP32 and FP64 mixed
        {"name": "serve_64", "kind": "serve", "count": 64, "spec": 11, "max_batch": 32},
    ]


# --------------------------------------------------------------------- draw

def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _is_smooth13(n: int) -> bool:
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _draw_length(rng, lo: int, hi: int) -> int:
    """Half powers of two, the rest 3*2^k / 5*2^k and other 13-smooth lengths."""
    u = rng.random()
    if u < 0.45:
        return 1 << rng.randint(math.ceil(math.log2(lo)), math.floor(math.log2(hi)))
    if u < 0.65:
        odd = rng.choice((3, 5))
        k = rng.randint(math.ceil(math.log2(lo / odd)), math.floor(math.log2(min(hi, 1 << 20) / odd)))
        return odd << k
    n = int(_log_uniform(rng, lo, min(hi, 1 << 20)))
    while not _is_smooth13(n):
        n -= 1
    return n


def draw(rng) -> dict:
    u = rng.random()
    bits = 32 if rng.random() < 0.65 else 64
    direction = FORWARD if rng.random() < 0.5 else BACKWARD
    if u < 0.08:
        return {"kind": "ragged", "count": int(_log_uniform(rng, 16, 512)),
                "spec": rng.randint(0, 999), "max_batch": rng.randint(4, 64)}
    if u < 0.14:
        return {"kind": "serve", "count": int(_log_uniform(rng, 8, 64)),
                "spec": rng.randint(0, 999), "max_batch": rng.randint(4, 32)}
    if u < 0.20:
        n = _draw_length(rng, 16, 1 << 18)
        return {"kind": "host", "n": n, "batch": max(1, int(_log_uniform(rng, 1 << 10, 1 << 21)) // n),
                "bits": bits, "direction": direction}
    if u < 0.30:
        n = _draw_length(rng, 16, 1 << 18)
        return {"kind": "fft", "n": n, "batch": max(1, int(_log_uniform(rng, 1 << 10, 1 << 24)) // n),
                "bits": bits, "direction": direction}
    kind = "filter" if u < 0.40 else "roundtrip" if u < 0.50 else "plan"
    n = _draw_length(rng, 16, 1 << (24 if kind == "plan" else 22))
    top = (1 << 26 if bits == 32 else 1 << 25) >> (0 if kind == "plan" else 1)
    return {"kind": kind, "n": n, "batch": max(1, int(_log_uniform(rng, 1 << 14, top)) // n),
            "bits": bits, "direction": direction}


# ------------------------------------------------------------------ prepare

_STREAM = None


def _stream() -> torch.cuda.Stream:
    """The program's stream: plans enqueue on it and return at once."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _dtype(case: dict):
    return torch.complex64 if case["bits"] == 32 else torch.complex128


def _uniform(shape, dtype, seed: int) -> torch.Tensor:
    """re / im iid uniform in [-1, 1)."""
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((*shape, 2), generator=g, device="cuda", dtype=real)
    return torch.view_as_complex(x.mul_(2).sub_(1))


def _host_uniform(case: dict, seed: int) -> np.ndarray:
    real = np.float32 if case["bits"] == 32 else np.float64
    v = np.random.default_rng(seed).random((case["batch"], case["n"], 2), dtype=real) * 2 - 1
    return v.view(np.complex64 if case["bits"] == 32 else np.complex128)[..., 0]


def _plan(case: dict, direction: int, placement: int = m.OUT_OF_PLACE) -> m.Plan:
    plan = m.Plan.create(case["n"], direction, placement, bits=case["bits"], batch=case["batch"])
    plan.set_stream(_stream().cuda_stream)
    return plan


def _all_pass(case: dict) -> torch.Tensor:
    """Unit-modulus transfer function (a quadratic phase) with the 1/n that
    unnormalised transforms leave to their caller."""
    n = case["n"]
    f = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
    h = torch.polar(torch.full_like(f, 1.0 / n), 40.0 * math.pi * f * f)
    return h.to(_dtype(case))


def _ragged_items(case: dict):
    return workloads.ragged_spec(case["count"], case["spec"], case["max_batch"])


def _serve_items(case: dict):
    return workloads.serving_stream(case["count"], 1.0, case["spec"], case["max_batch"])


def _serve_arenas(case: dict, seed: int):
    """Input arenas per precision and every request with its offset in them."""
    points = {32: 0, 64: 0}
    placed = []
    for r in _serve_items(case):
        placed.append((r, points[r["bits"]]))
        points[r["bits"]] += r["n"] * r["batch"]
    arenas = {b: _uniform((max(1, p),), torch.complex64 if b == 32 else torch.complex128, seed + b)
              for b, p in points.items()}
    return placed, arenas


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = {"kind": kind, "direction": case.get("direction")}
    if kind == "ragged":
        items = _ragged_items(case)
        x = _uniform((sum(n * b for n, b, _ in items),), torch.complex64, seed)
        y = torch.empty_like(x)
        views, at = [], 0
        for n, b, d in items:
            views.append((x[at:at + n * b].view(b, n), y[at:at + n * b].view(b, n), d))
            at += n * b
        s.update(x=x, y=y, plan=m.RaggedPlan(views), stream=_stream().cuda_stream)
    elif kind == "serve":
        placed, xs = _serve_arenas(case, seed)
        ys = {b: torch.zeros_like(x) for b, x in xs.items()}
        requests = []
        for r, at in placed:
            step = xs[r["bits"]].element_size()
            requests.append((r["n"], r["batch"], r["direction"], r["bits"],
                             xs[r["bits"]].data_ptr() + at * step,
                             ys[r["bits"]].data_ptr() + at * step))
        server = m.Server()
        s.update(xs=xs, ys=ys, requests=requests, server=server)
    elif kind == "host":
        x = _host_uniform(case, seed)
        plan = m.Plan.create(case["n"], case["direction"], bits=case["bits"], batch=case["batch"])
        s.update(x=x, y=np.empty_like(x), plan=plan)
    else:
        x = _uniform((case["batch"], case["n"]), _dtype(case), seed)
        s["x"] = x
        if kind == "filter":
            s.update(fwd=_plan(case, FORWARD, m.IN_PLACE), bwd=_plan(case, BACKWARD, m.IN_PLACE),
                     h=_all_pass(case), stream=_stream())
        elif kind == "roundtrip":
            s.update(fwd=_plan(case, FORWARD), bwd=_plan(case, BACKWARD),
                     y=torch.empty_like(x), z=torch.empty_like(x))
        elif kind == "plan":
            s.update(plan=_plan(case, case["direction"]), y=torch.empty_like(x))
    return s


# ---------------------------------------------------------------------- run

def run(s: dict):
    kind = s["kind"]
    if kind == "plan":
        s["plan"].execute(s["x"], s["y"])
        return s["y"]
    if kind == "fft":
        return m.fft(s["x"], s["direction"])
    if kind == "host":
        s["plan"].execute(s["x"], s["y"])
        return s["y"]
    if kind == "roundtrip":
        s["fwd"].execute(s["x"], s["y"])
        s["bwd"].execute(s["y"], s["z"])
        return [s["y"], s["z"]]
    if kind == "filter":
        x = s["x"]
        s["fwd"].execute(x)
        with torch.cuda.stream(s["stream"]):
            x.mul_(s["h"])
        s["bwd"].execute(x)
        return x
    if kind == "ragged":
        s["plan"].execute(s["stream"])
        return s["y"]
    server = s["server"]
    for request in s["requests"]:
        server.submit(*request)
    server.drain()
    return [s["ys"][32], s["ys"][64]]


# --------------------------------------------------------------------- work

def work(case: dict) -> dict:
    """Every input read once, every output written once; 5 n log2 n flops."""
    kind = case["kind"]
    if kind in ("ragged", "serve"):
        if kind == "ragged":
            items = [(n, b, 32) for n, b, _ in _ragged_items(case)]
        else:
            items = [(r["n"], r["batch"], r["bits"]) for r in _serve_items(case)]
        return {"bytes": sum(n * b * bits // 2 for n, b, bits in items),
                "flops": sum(5 * n * b * math.log2(n) for n, b, _ in items)}
    n, points = case["n"], case["n"] * case["batch"]
    value = case["bits"] // 4
    flops = 5 * points * math.log2(n)
    if kind == "roundtrip":
        return {"bytes": 3 * points * value, "flops": 2 * flops}
    if kind == "filter":
        return {"bytes": 2 * points * value + n * value, "flops": 2 * flops + 6 * points}
    return {"bytes": 2 * points * value, "flops": flops}


# -------------------------------------------------------------------- exact

def _dft(x: torch.Tensor, direction: int) -> torch.Tensor:
    x = x.to(torch.complex128)
    return torch.fft.fft(x) if direction == FORWARD else torch.fft.ifft(x, norm="forward")


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "host":
        x = _host_uniform(case, seed).astype(np.complex128)
        if case["direction"] == FORWARD:
            return np.fft.fft(x)
        return np.fft.ifft(x, norm="forward")
    if kind == "ragged":
        items = _ragged_items(case)
        x = _uniform((sum(n * b for n, b, _ in items),), torch.complex64, seed)
        out, at = torch.empty(x.shape, dtype=torch.complex128, device="cuda"), 0
        for n, b, d in items:
            out[at:at + n * b] = _dft(x[at:at + n * b].view(b, n), d).view(-1)
            at += n * b
        return out
    if kind == "serve":
        placed, xs = _serve_arenas(case, seed)
        outs = {b: torch.zeros(x.shape, dtype=torch.complex128, device="cuda")
                for b, x in xs.items()}
        for r, at in placed:
            n, b = r["n"], r["batch"]
            part = xs[r["bits"]][at:at + n * b].view(b, n)
            outs[r["bits"]][at:at + n * b] = _dft(part, r["direction"]).view(-1)
        return [outs[32], outs[64]]
    x = _uniform((case["batch"], case["n"]), _dtype(case), seed)
    if kind == "roundtrip":
        return [_dft(x, FORWARD), x.to(torch.complex128) * case["n"]]
    if kind == "filter":
        h = _all_pass(case).to(torch.complex128)
        return _dft(_dft(x, FORWARD) * h, BACKWARD)
    return _dft(x, case["direction"])
