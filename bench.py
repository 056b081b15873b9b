#!/usr/bin/env python
"""Benchmark of the PencilFFTs transform path on GB300.

Workload (the reference's headline benchmark, benchmarks/benchmarks.jl:200-266,
at one GPU): a 3D Float64 RFFT plan on a 512^3 grid, permute_dims=true,
out-of-place; one step = ``mul!(v, plan, u)`` followed by ``ldiv!(u, plan, v)``
(a forward r2c + backward c2r round trip, the scaling fused in the last pass).
Input: uniform [-1, 1), seeded.  Every array is far larger than L2 (1.07 GB).

Prints one JSON line.  ``--impl reference`` times the CPU oracle (the
restatement of the reference path with scipy.fft, all host cores) on the same
workload instead.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import tempfile
import sys
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
for _p in (REPO, os.path.join(REPO, "pencilffts.jl_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

METRIC = "512^3 r2c+c2r round-trip ms"
UNIT = "ms"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--dims", default="512,512,512")
    ap.add_argument("--real", default="f64", choices=["f64", "f32"])
    ap.add_argument("--precision", default="default", choices=["default", "native", "fx", "tc"])
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-forms", action="store_true",
                    help="skip the Float32 plain vs tensor-core split comparison")
    ap.add_argument("--cpu-sample-s", type=float, default=20.0,
                    help="approximate CPU seconds for the cpu_baseline sample")
    ap.add_argument("--configs", default="all",
                    help="other benchmark configurations to measure after the headline: "
                         "'all', 'none' or a comma list of C1,C2a,C2b,C3,C4,C5,long_lines")
    ap.add_argument("--config-steps", type=int, default=10)
    ap.add_argument("--profile-batch", action="store_true",
                    help="for ncu: build the 64 uneven Float32 fields of configuration C5, launch the batch "
                         "once in the persistent form and once in the graph form, and exit")
    return ap.parse_args()


def workload(args):
    dims = tuple(int(x) for x in args.dims.split(","))
    rb = 8 if args.real == "f64" else 4
    return dims, rb


ARITHMETIC = {
    ("f64", "default"): "int32 + FP32 pairs in the butterflies, dd (2xFP32, 48-bit significand) around them",
    ("f64", "native"): "FP64",
    ("f64", "fx"): "block floating point (int64 components, per-line exponent)",
    ("f32", "default"): "FP32",
    ("f32", "tc"): "FP32 with 3xTF32 tensor-core DFT products for 256/512/1024-point c2c lines",
}


def headline_config(args, world):
    """The workload description both arms print (identical dicts)."""
    dims, rb = workload(args)
    arith = ARITHMETIC.get((args.real, args.precision), args.precision)
    return {"workload": f"RFFT round trip {'x'.join(map(str, dims))} "
                        f"{'Float64' if rb == 8 else 'Float32'} (mul! + ldiv!), "
                        "permute_dims=true, out-of-place",
            "dims": list(dims), "transforms": "RFFT (RFFT, FFT, FFT)",
            "l2": (f"inputs larger than L2 ({int(np.prod(dims)) * rb / 1e9:.2f} GB arrays)"
                   if int(np.prod(dims)) * rb > 129e6 else "inputs L2-resident (smaller than 129 MB)"),
            "precision": f"{'Float64' if rb == 8 else 'Float32'} data; GB300 arm: {arith}; "
                         "reference arm: FP64 (oracle, scipy.fft)",
            "parallelism": f"replicas x{world}" if world > 1 else "single GPU"}


def alg_bytes_round_trip(dims, rb):
    """One read + one write per pass: forward R + C + 2C*(N-1)... for a 3D r2c
    this is R + 5C per direction (2(R + 5C) per round trip)."""
    import numpy as np
    n = int(np.prod(dims))
    R = n * rb
    C = (dims[0] // 2 + 1) * int(np.prod(dims[1:])) * 2 * rb
    N = len(dims)
    per_dir = (R + C) + 2 * C * (N - 1)
    return 2 * per_dir, R, C


# ---------------------------------------------------------------------------
# CPU oracle timing (cpu_baseline and the reference arm)
# ---------------------------------------------------------------------------
def time_cpu_oracle(dims, rb, budget_s, max_iters=None):
    """Times the oracle's forward + ldiv (scipy.fft, all host threads) on the
    full workload; returns (ms per round trip, iterations, threads)."""
    import numpy as np
    import scipy.fft as sfft
    from oracle import pencilfft_oracle as O

    threads = os.cpu_count() or 1
    real = np.float64 if rb == 8 else np.float32
    rng = np.random.default_rng(1)
    u = rng.uniform(-1.0, 1.0, size=dims).astype(real)
    plan = O.OraclePlan(dims, O.RFFT(), real)
    times = []
    t_start = time.perf_counter()
    with sfft.set_workers(threads):
        while True:
            t0 = time.perf_counter()
            v = plan.forward(u)
            u2 = plan.ldiv(v)
            times.append(time.perf_counter() - t0)
            del v, u2
            if max_iters is not None and len(times) >= max_iters:
                break
            if max_iters is None and time.perf_counter() - t_start >= budget_s:
                break
    return 1e3 * statistics.mean(times), len(times), threads


def max_over_ranks(value: float, world: int, device=None) -> float:
    """Max of a per-rank timing over all ranks (the slowest replica sets the
    step time); identity at one rank."""
    if world <= 1:
        return float(value)
    import torch
    import torch.distributed as dist
    t = torch.tensor([float(value)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ---------------------------------------------------------------------------
# clocks sampled during the timed region
# ---------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        # raw samples (the JSON line carries their summary); PFGB_CLOCKS_DIR
        # keeps them in a chosen folder
        self.path = os.path.join(os.environ.get("PFGB_CLOCKS_DIR", tempfile.gettempdir()),
                                 f"clocks_bench_{os.getpid()}.csv")

    def start(self):
        try:
            os.makedirs(os.path.dirname(self.path), exist_ok=True)
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.f.close()
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                rows.append(parts)
            except ValueError:
                pass
        if not rows:
            return None
        sm = [float(r[1]) for r in rows if r[1].replace(".", "", 1).isdigit()]
        smax = [float(r[2]) for r in rows if r[2].replace(".", "", 1).isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in rows:
            for i, nm in enumerate(names):
                if r[5 + i].lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(rows)}


# ---------------------------------------------------------------------------
# Float32 forms: plain path against the tensor-core split form
# ---------------------------------------------------------------------------
def measure_forms(P, dims, steps, warmup, dev):
    """Times the Float32 RFFT round trip of the same workload with the plain
    kernels and with the tensor-core split form (precision="tc"), and states
    each form's error: rel. L2 of the forward spectrum against the Float64
    plan's spectrum (the double-float path, parity-tested against the FP64
    oracle at 1e-13) and of the round trip against the input."""
    import numpy as np
    import torch

    T = P.Transforms
    g = torch.Generator(device=dev)
    g.manual_seed(7)
    p64 = P.PencilFFTPlan(dims, T.RFFT(), np.float64)
    u64 = p64.allocate_input()
    u64.data.uniform_(-1.0, 1.0, generator=g)
    ref = p64 * u64
    ref_norm = torch.linalg.vector_norm(ref.data).item()
    stream = torch.cuda.current_stream()
    out = {}
    for name, prec in (("f32_plain", "default"), ("f32_tc_split", "tc")):
        p = P.PencilFFTPlan(dims, T.RFFT(), np.float32, precision=prec)
        u, v, w = p.allocate_input(), p.allocate_output(), p.allocate_input()
        u.data.copy_(u64.data)
        P.mul_(v, p, u)
        e_fwd = (torch.linalg.vector_norm(v.data.to(ref.data.dtype) - ref.data).item() / ref_norm)
        P.ldiv_(w, p, v)
        e_rt = (torch.linalg.vector_norm(w.data - u.data).item() / torch.linalg.vector_norm(u.data).item())
        for _ in range(warmup):
            P.mul_(v, p, u)
            P.ldiv_(w, p, v)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(steps):
            P.mul_(v, p, u)
            P.ldiv_(w, p, v)
        e1.record(stream)
        torch.cuda.synchronize()
        out[name] = {"value": e0.elapsed_time(e1) / steps, "unit": UNIT,
                     "rel_l2_forward": e_fwd, "rel_l2_round_trip": e_rt}
        del p, u, v, w
        torch.cuda.empty_cache()
    out["tc_split_speedup_vs_plain"] = out["f32_plain"]["value"] / out["f32_tc_split"]["value"]
    out["error_reference"] = ("forward: Float64 plan on the same input (double-float path, "
                              "parity-tested against the FP64 oracle at 1e-13); round trip: the input")
    del p64, u64, ref
    torch.cuda.empty_cache()
    return out


# ---------------------------------------------------------------------------
# The other benchmark configurations (C1-C5).  Each is timed on the device as
# mul! + ldiv! per step (the reference benchmark loop), with the dominant
# kernel's roofline from per-pass events; its CPU leg times the oracle on the
# same input and, as the checker, gives the forward rel. L2 of the GPU output
# against it.
# ---------------------------------------------------------------------------
def _rel(a, b, chunk=1 << 24):
    """|a - b| / |b| in float64 over chunks (host arrays)."""
    import numpy as np
    a = np.asarray(a).reshape(-1)
    b = np.asarray(b).reshape(-1)
    num = den = 0.0
    for i in range(0, a.size, chunk):
        x, y = a[i:i + chunk], b[i:i + chunk]
        num += float(np.sum(np.abs(x.astype(np.complex128) - y) ** 2))
        den += float(np.sum(np.abs(y) ** 2))
    return (num / den) ** 0.5 if den > 0 else num ** 0.5


def _rel_dev(a, b):
    """|a - b| / |b| on the device, in float64."""
    import torch
    a = torch.view_as_real(a) if a.is_complex() else a
    b = torch.view_as_real(b) if b.is_complex() else b
    return (torch.linalg.vector_norm((a.double() - b.double()).reshape(-1)) /
            torch.linalg.vector_norm(b.double().reshape(-1))).item()


def _peak():
    try:
        return float(json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def _roofline(timing, steps):
    """Dominant kernel (largest summed event time) of the per-pass records of
    `steps` timed steps: algorithmic bytes per launch / average duration."""
    per = {}
    for e in timing:
        k = per.setdefault(e["kernel"], {"ms": 0.0, "bytes": 0, "launches": 0})
        k["ms"] += e["total_ms"]
        k["bytes"] += e["bytes_per_launch"] * e["launches"]
        k["launches"] += e["launches"]
    name, d = max(per.items(), key=lambda kv: kv[1]["ms"])
    peak, src = _peak()
    bpl = d["bytes"] / d["launches"]
    avg_s = d["ms"] / d["launches"] * 1e-3
    ach = bpl / avg_s / 1e9
    return {"bound": "hbm", "kernel": name, "achieved": ach, "peak": peak, "peak_source": src,
            "unit": "GB/s", "frac": ach / peak, "alg_bytes_per_launch": bpl,
            "avg_launch_ms": avg_s * 1e3, "launches_per_step": sum(v["launches"] for v in per.values()) / steps,
            "kernel_share": d["ms"] / sum(v["ms"] for v in per.values())}


def _timed(steps, warmup, step, plans=(), stats=None):
    """ms per step (CUDA events on the current stream, synchronised on both
    sides) and the plans' per-pass records of the timed steps; `stats`, when
    given, receives the mean, std, min and max of the steps (one event
    between consecutive steps)."""
    import numpy as np
    import torch
    for _ in range(warmup):
        step()
    torch.cuda.synchronize()
    for p in plans:
        p.set_timing(True)
    stream = torch.cuda.current_stream()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
    evs[0].record(stream)
    for i in range(steps):
        step()
        evs[i + 1].record(stream)
    torch.cuda.synchronize()
    timing = []
    for p in plans:
        timing += p.get_timing()
        p.set_timing(False)
    if stats is not None:
        per = np.array([evs[i].elapsed_time(evs[i + 1]) for i in range(steps)])
        stats.update(mean=float(per.mean()), std=float(per.std()), min=float(per.min()),
                     max=float(per.max()), n=int(steps))
    return evs[0].elapsed_time(evs[-1]) / steps, timing


def _kernels(timing, steps):
    """Per kernel of the timed steps: device ms per step, launches per step and
    algorithmic GB/s (one read of each pass input + one write of its output)."""
    per = {}
    for e in timing:
        k = per.setdefault(e["kernel"], {"ms": 0.0, "bytes": 0, "launches": 0})
        k["ms"] += e["total_ms"]
        k["bytes"] += e["bytes_per_launch"] * e["launches"]
        k["launches"] += e["launches"]
    return {name: {"ms_per_step": d["ms"] / steps, "launches_per_step": d["launches"] / steps,
                   "gbs": d["bytes"] / (d["ms"] * 1e-3) / 1e9 if d["ms"] > 0 else None}
            for name, d in sorted(per.items(), key=lambda kv: -kv[1]["ms"])}


def _oracle_leg(forward, x, got):
    """cpu_baseline leg of a configuration: the oracle's forward transform of
    the same input, timed on the host threads, and (as the checker) the rel.
    L2 of the GPU forward output against it."""
    t0 = time.perf_counter()
    ref = forward(x)
    ms = (time.perf_counter() - t0) * 1e3
    return ms, _rel(got, ref)


def _round_trip_config(P, O, steps, warmup, dims, transforms, real, x, workload, data, gflop=None):
    import numpy as np
    import torch
    plan = P.PencilFFTPlan(dims, transforms, real)
    u, v, w = plan.allocate_input(), plan.allocate_output(), plan.allocate_input()
    u.copy_from_logical(x)

    def step():
        P.mul_(v, plan, u)
        P.ldiv_(w, plan, v)

    stats = {}
    ms, timing = _timed(steps, warmup, step, (plan,), stats)
    alg = sum(e["bytes_per_launch"] * e["launches"] for e in timing) / steps
    P.mul_(v, plan, u)
    P.ldiv_(w, plan, v)
    got, back = v.to_logical(), w.to_logical()
    orc = O.OraclePlan(dims, tuple(_to_oracle(O, P, t) for t in plan.transforms), np.dtype(real))
    threads = os.cpu_count() or 1
    import scipy.fft as sfft
    with sfft.set_workers(threads):
        fwd_ms, err = _oracle_leg(orc.forward, x, got)
    out = {"workload": workload, "data": data, "dims": list(dims),
           "value": ms, "unit": "ms", "metric": "round trip (mul! + ldiv!) ms", "step_ms": stats,
           "forward_ms": sum(e["total_ms"] for e in timing if e["direction"] > 0) / steps,
           "backward_ms": sum(e["total_ms"] for e in timing if e["direction"] < 0) / steps,
           "alg_bytes_per_round_trip": alg, "hbm_gbs": alg / (ms * 1e-3) / 1e9,
           "roofline": _roofline(timing, steps), "kernels": _kernels(timing, steps),
           "rel_l2_forward_vs_oracle": err, "rel_l2_round_trip": _rel(back, x),
           "cpu_baseline": {"value": fwd_ms, "unit": "ms per forward", "cores": threads, "kind": "port",
                            "sample": "one forward transform of the same input (oracle, scipy.fft)"}}
    if gflop is not None:
        out["gflops"] = gflop / (ms * 1e-3)
    del plan, u, v, w
    torch.cuda.empty_cache()
    return out


def _to_oracle(O, P, tr):
    T = P.Transforms
    if isinstance(tr, T.FFT):
        return O.Tr("FFT", tr.inplace)
    if isinstance(tr, T.BFFT):
        return O.Tr("BFFT", tr.inplace)
    if isinstance(tr, T.RFFT):
        return O.Tr("RFFT", tr.inplace)
    if isinstance(tr, T.BRFFT):
        return O.Tr("BRFFT", tr.inplace, even=tr.even_output)
    if isinstance(tr, T.R2R):
        return O.Tr("R2R", tr.inplace, kind=tr.kind)
    return O.Tr("NoTransform", tr.inplace)


def _flop_c2c(n):
    import numpy as np
    return 2 * 5 * n * np.log2(n) / 1e9  # forward + backward, 5 N log2 N each


def _flop_r2c(n):
    import numpy as np
    return 2 * 2.5 * n * np.log2(n) / 1e9


def config_c1(P, O, steps, warmup):
    import numpy as np
    dims = (16, 32, 64)
    x = np.random.default_rng(42).random(dims)
    return _round_trip_config(P, O, steps, warmup, dims, P.Transforms.RFFT(), np.float64, x,
                              "RFFT round trip 16x32x64 Float64", "uniform [0,1), seed 42 (L2-resident)",
                              _flop_r2c(np.prod(dims)))


def config_c2a(P, O, steps, warmup):
    import numpy as np
    dims = (256, 256, 256)
    rng = np.random.default_rng(0)
    x = rng.standard_normal(dims) + 1j * rng.standard_normal(dims)
    return _round_trip_config(P, O, steps, warmup, dims, P.Transforms.FFT(), np.float64, x,
                              "FFT + BFFT (ldiv!) round trip 256^3 ComplexF64",
                              "N(0,1) real and imaginary parts, seed 0 (268 MB arrays)",
                              _flop_c2c(np.prod(dims)))


def config_c2b(P, O, steps, warmup):
    import numpy as np
    dims = (512, 512, 512)
    x = np.random.default_rng(1).uniform(-1, 1, dims).astype(np.float32)
    return _round_trip_config(P, O, steps, warmup, dims, P.Transforms.RFFT(), np.float32, x,
                              "RFFT round trip 512^3 Float32", "uniform [-1,1), seed 1 (537 MB arrays)",
                              _flop_r2c(np.prod(dims)))


def config_c3(P, O, steps, warmup):
    import numpy as np
    T = P.Transforms
    nx, ny, nz = 512, 512, 257
    xs = 2 * np.pi * np.arange(nx) / nx
    ys = 2 * np.pi * np.arange(ny) / ny
    zs = np.cos(np.pi * np.arange(nz) / (nz - 1))
    u = np.sin(xs)[:, None, None] * np.cos(ys)[None, :, None] * np.cos(zs)[None, None, :]
    return _round_trip_config(P, O, steps, warmup, (nx, ny, nz), (T.RFFT(), T.FFT(), T.R2R(T.REDFT00)),
                              np.float64, u,
                              "(RFFT, FFT, R2R{REDFT00}) round trip 512x512x257 Float64",
                              "Taylor-Green sin x cos y cos z, Chebyshev-Gauss-Lobatto z (539 MB arrays)",
                              _flop_r2c(512 ** 3))


def config_c4(P, O, steps, warmup):
    """1024^3 Float32 RFFT, plain and tensor-core split form; errors against
    the Float64 plan on the same input (the double-float path, itself
    parity-tested against the FP64 oracle at 1e-13; a 1024^3 CPU oracle per
    run is too slow)."""
    import numpy as np
    import torch
    n = 1024
    dims = (n, n, n)
    T = P.Transforms
    rng = np.random.default_rng(1234)
    amps, phis, ks = rng.uniform(1, 10, 8), rng.uniform(0, 2 * np.pi, 8), rng.integers(0, 64, size=(8, 3))
    p64 = P.PencilFFTPlan(dims, T.RFFT(), np.float64)
    u64 = p64.allocate_input()
    g = torch.Generator(device="cuda").manual_seed(1234)
    u64.data.normal_(generator=g)
    lin = torch.arange(n, device="cuda", dtype=torch.float64) * (2 * np.pi / n)
    for a, phi, k in zip(amps, phis, ks):
        ph = (k[2] * lin)[:, None, None] + (k[1] * lin)[None, :, None] + (k[0] * lin)[None, None, :]
        u64.data.add_(a * torch.cos(ph + phi))
        del ph
    u64.data.copy_(u64.data.float().double())  # the Float32 input, exactly
    ref = p64 * u64
    del p64
    torch.cuda.empty_cache()
    out = {"workload": "RFFT round trip 1024^3 Float32, plain and tensor-core split forms",
           "data": "N(0,1) + 8 random-amplitude Fourier modes, seed 1234 (4.3 GB arrays)", "dims": list(dims)}
    for name, prec in (("f32_plain", "default"), ("f32_tc_split", "tc")):
        p = P.PencilFFTPlan(dims, T.RFFT(), np.float32, precision=prec)
        u, v, w = p.allocate_input(), p.allocate_output(), p.allocate_input()
        u.data.copy_(u64.data)

        def step():
            P.mul_(v, p, u)
            P.ldiv_(w, p, v)

        ms, timing = _timed(steps, warmup, step, (p,))
        alg = sum(e["bytes_per_launch"] * e["launches"] for e in timing) / steps
        P.mul_(v, p, u)
        P.ldiv_(w, p, v)
        out[name] = {"value": ms, "unit": "ms", "hbm_gbs": alg / (ms * 1e-3) / 1e9,
                     "gflops": _flop_r2c(n ** 3) / (ms * 1e-3), "roofline": _roofline(timing, steps),
                     "rel_l2_forward_vs_f64": _rel_dev(v.data, ref.data),
                     "rel_l2_round_trip": _rel_dev(w.data, u.data),
                     "device_status": p.device_status()}
        del p, u, v, w
        torch.cuda.empty_cache()
    out["tc_split_speedup_vs_plain"] = out["f32_plain"]["value"] / out["f32_tc_split"]["value"]
    del u64, ref
    torch.cuda.empty_cache()
    return out


def config_c5(P, O, steps, warmup):
    """(i) 3 x 384^3 Float32: per component c, r2c, i k_c multiply fused into
    the first backward pass, c2r (the derivative along dimension c);
    (ii) 64 independent r2c/c2r round trips of sizes drawn from 48..192 per
    axis, recorded once into a CUDA graph (Batch) and replayed."""
    import numpy as np
    import scipy.fft as sfft
    import torch
    T = P.Transforms
    threads = os.cpu_count() or 1
    out = {}
    # (i) vector field
    n = 384
    dims = (n, n, n)
    plan = P.PencilFFTPlan(dims, T.RFFT(), np.float32)
    rng = np.random.default_rng(2024)
    comps = [rng.standard_normal(dims).astype(np.float32) for _ in range(3)]
    us = plan.allocate_input(P.Val(3))
    vs = plan.allocate_output(P.Val(3))
    ds = plan.allocate_input(P.Val(3))
    for c, x in zip(us, comps):
        c.copy_from_logical(x)
    L = 2 * np.pi

    def step():
        for c in range(3):
            P.mul_(vs[c], plan, us[c])
            P.ldiv_(ds[c], plan, vs[c], deriv=(c + 1, L))

    ms, timing = _timed(steps, warmup, step, (plan,))
    alg = sum(e["bytes_per_launch"] * e["launches"] for e in timing) / steps
    step()
    orc = O.OraclePlan(dims, O.RFFT(), np.float32)
    errs = []
    t0 = time.perf_counter()
    with sfft.set_workers(threads):
        for c in range(3):
            ref = orc.ldiv(orc.forward(comps[c]) * O.wavenumbers(orc, c, L))
            errs.append(_rel(ds[c].to_logical(), ref))
    cpu_ms = (time.perf_counter() - t0) * 1e3
    out["vector_gradient_384"] = {
        "workload": "3 x 384^3 Float32: r2c, i k_c fused into the first backward pass, c2r (per component)",
        "data": "N(0,1), seed 2024 (227 MB per component)", "value": ms, "unit": "ms per 3 components",
        "hbm_gbs": alg / (ms * 1e-3) / 1e9, "roofline": _roofline(timing, steps),
        "rel_l2_vs_oracle_max": max(errs),
        "cpu_baseline": {"value": cpu_ms, "unit": "ms per 3 components", "cores": threads, "kind": "port",
                         "sample": "oracle forward, i k multiply and ldiv of the 3 components"}}
    del plan, us, vs, ds
    torch.cuda.empty_cache()
    # (ii) 64 uneven fields
    rng = np.random.default_rng(2024)
    sizes = [tuple(int(s) for s in rng.integers(48, 193, 3)) for _ in range(64)]
    plans, arrs, xs = [], [], []
    for d in sizes:
        p = P.PencilFFTPlan(d, T.RFFT(), np.float32)
        u, v, w = p.allocate_input(), p.allocate_output(), p.allocate_input()
        x = rng.standard_normal(d).astype(np.float32)
        u.copy_from_logical(x)
        plans.append(p)
        arrs.append((u, v, w))
        xs.append(x)
    alg = 0
    for p, (u, v, w) in zip(plans, arrs):
        _, t = _timed(1, 0, lambda: (P.mul_(v, p, u), P.ldiv_(w, p, v)), (p,))
        alg += sum(e["bytes_per_launch"] * e["launches"] for e in t)

    def seq():
        for p, (u, v, w) in zip(plans, arrs):
            P.mul_(v, p, u)
            P.ldiv_(w, p, v)

    ms_seq, _ = _timed(steps, warmup, seq)
    ops = []
    for p, (u, v, w) in zip(plans, arrs):
        ops += [(P.mul_, v, p, u), (P.ldiv_, w, p, v)]
    graph = P.Batch(ops, form="graph")
    ms_graph, _ = _timed(steps, warmup, graph.launch)
    del graph
    pers = P.Batch(ops, form="persistent")
    pinfo = pers.info()
    ms_pers, _ = _timed(steps, warmup, pers.launch)
    del pers
    # the batch autotuner: both forms (and the persistent list's orders) timed
    # at creation, the fastest kept
    batch = P.Batch(ops, form="measure")
    binfo = batch.info()
    ms_best, _ = _timed(steps, warmup, batch.launch)
    batch.launch()
    torch.cuda.synchronize()
    errs, rts = [], []
    t0 = time.perf_counter()
    for p, (u, v, w), x, d in zip(plans, arrs, xs, sizes):
        o = O.OraclePlan(d, O.RFFT(), np.float32)
        errs.append(_rel(v.to_logical(), o.forward(x)))
        rts.append(_rel(w.to_logical(), x))
    cpu_ms = (time.perf_counter() - t0) * 1e3
    out["uneven_64"] = {
        "workload": "64 independent r2c + c2r round trips, sizes ~U{48..192} per axis (seed 2024), "
                    "one batch launch in the form the batch autotuner kept",
        "data": "N(0,1) (fields of 0.4-28 MB, L2-resident)", "value": ms_best, "unit": "ms per 64 round trips",
        "form": binfo["form"], "graph_form_ms": ms_graph, "persistent_form_ms": ms_pers,
        "sequential_ms": ms_seq, "speedup_vs_sequential": ms_seq / ms_best,
        "autotuner_measured": {"graph_ms": binfo["graph_ms"], "persistent_best_order_ms": binfo["persistent_ms"]},
        "persistent_work_list": {k: pinfo[k] for k in ("items", "tiles", "grid", "smem", "wave_bytes")},
        "hbm_gbs": alg / (ms_best * 1e-3) / 1e9, "alg_bytes": alg,
        "rel_l2_forward_vs_oracle_max": max(errs), "rel_l2_round_trip_max": max(rts),
        "cpu_baseline": {"value": cpu_ms, "unit": "ms (oracle forwards of the 64 fields, checker included)",
                         "cores": 1, "kind": "port", "sample": "one forward per field"}}
    del batch
    # (iii) the whole set in one persistent launch: the 3-component gradient
    # of (i) and the 64 fields of (ii)
    n = 384
    vplan = P.PencilFFTPlan((n, n, n), T.RFFT(), np.float32)
    us = vplan.allocate_input(P.Val(3))
    vs = vplan.allocate_output(P.Val(3))
    ds = vplan.allocate_input(P.Val(3))
    rng = np.random.default_rng(2024)
    for c in us:
        c.copy_from_logical(rng.standard_normal((n, n, n)).astype(np.float32))
    gops = []
    for c in range(3):
        gops += [(P.mul_, vs[c], vplan, us[c]), (P.ldiv_, ds[c], vplan, vs[c], (c + 1, 2 * np.pi))]
    ms_parts = {}
    for name, o in (("gradient", gops), ("uneven", ops)):
        b = P.Batch(o, form="persistent")
        ms_parts[name], _ = _timed(steps, warmup, b.launch)
        del b
    allb = P.Batch(gops + ops, form="persistent")
    ainfo = allb.info()
    ms_all, _ = _timed(steps, warmup, allb.launch)
    del allb
    allg = P.Batch(gops + ops, form="graph")
    ms_allg, _ = _timed(steps, warmup, allg.launch)
    del allg
    out["c5_one_launch"] = {
        "workload": "3 x 384^3 Float32 spectral gradient (i k_c fused) + the 64 uneven round trips, "
                    "one persistent launch",
        "value": ms_all, "unit": "ms per launch", "graph_form_ms": ms_allg,
        "gradient_alone_persistent_ms": ms_parts["gradient"], "uneven_alone_persistent_ms": ms_parts["uneven"],
        "work_list": {k: ainfo[k] for k in ("items", "tiles", "grid", "smem", "wave_bytes")}}
    del plans, arrs, vplan, us, vs, ds
    torch.cuda.empty_cache()
    # (iv) many small fields, the launch-bound regime of the batched form:
    # 256 r2c + c2r round trips of 16^3
    plans, arrs, ops = [], [], []
    for _ in range(256):
        p = P.PencilFFTPlan((16, 16, 16), T.RFFT(), np.float32)
        u, v, w = p.allocate_input(), p.allocate_output(), p.allocate_input()
        u.copy_from_logical(rng.standard_normal((16, 16, 16)).astype(np.float32))
        plans.append(p)
        arrs.append((u, v, w))
        ops += [(P.mul_, v, p, u), (P.ldiv_, w, p, v)]
    forms = {}
    for f in ("graph", "persistent", "measure"):
        b = P.Batch(ops, form=f)
        forms[f], _ = _timed(steps, warmup, b.launch)
        if f == "measure":
            kept = b.form
        del b
    ms_seq_small, _ = _timed(steps, warmup, lambda: [(P.mul_(v, p, u), P.ldiv_(w, p, v))
                                                       for p, (u, v, w) in zip(plans, arrs)])
    out["small_fields_256"] = {
        "workload": "256 independent r2c + c2r round trips of 16^3 Float32 (launch-bound batch)",
        "value": forms["measure"], "unit": "ms per 256 round trips", "form": kept,
        "graph_form_ms": forms["graph"], "persistent_form_ms": forms["persistent"],
        "sequential_ms": ms_seq_small}
    del plans, arrs, ops
    torch.cuda.empty_cache()
    return out


def config_long_lines(P, O, steps, warmup):
    """Lines beyond one register pass: a long r2c axis (packed pair of real
    lines, split c2c transform, separating map) and a prime c2c length
    (Bluestein convolution through split power-of-two transforms)."""
    import numpy as np
    rng = np.random.default_rng(11)
    dims = (16384, 4096)
    x = rng.standard_normal(dims)
    out = {"rfft_16384x4096_f64": _round_trip_config(
        P, O, steps, warmup, dims, P.Transforms.RFFT(), np.float64, x,
        "RFFT round trip 16384x4096 Float64 (16384-point r2c lines)", "N(0,1), seed 11 (537 MB arrays)",
        _flop_r2c(np.prod(dims)))}
    dims = (8209, 1024)
    x = rng.standard_normal(dims) + 1j * rng.standard_normal(dims)
    out["fft_8209x1024_f64"] = _round_trip_config(
        P, O, steps, warmup, dims, P.Transforms.FFT(), np.float64, x,
        "FFT + BFFT round trip 8209x1024 ComplexF64 (prime 8209-point lines, Bluestein)",
        "N(0,1) real and imaginary parts, seed 11 (134 MB arrays)", _flop_c2c(np.prod(dims)))
    return out


CONFIGS = {"C1": config_c1, "C2a": config_c2a, "C2b": config_c2b, "C3": config_c3,
           "C4": config_c4, "C5": config_c5, "long_lines": config_long_lines}


# ---------------------------------------------------------------------------
# the GB300 arm
# ---------------------------------------------------------------------------
def run_gpu(args, rank, world, local_rank):
    import numpy as np
    import torch
    import torch.distributed as dist

    import pencilffts_gb300 as P

    dims, rb = workload(args)
    real = np.float64 if rb == 8 else np.float32
    T = P.Transforms

    # CPU baseline first (host threads only, before any GPU work of this rank)
    cpu_baseline = None
    if rank == 0 and not args.no_cpu_baseline:
        ms, iters, threads = time_cpu_oracle(dims, rb, args.cpu_sample_s)
        cpu_baseline = {"value": ms, "unit": UNIT, "cores": threads, "kind": "port",
                        "sample": f"{iters} full {'x'.join(map(str, dims))} "
                                  f"{'Float64' if rb == 8 else 'Float32'} RFFT round trips "
                                  f"(oracle: scipy.fft pocketfft, {threads} threads; Julia and "
                                  "FFTW are not installed, so the reference's FFTW path is "
                                  "replaced by this restatement)"}

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    plan = P.PencilFFTPlan(dims, T.RFFT(), real, precision=args.precision)
    u = plan.allocate_input()
    v = plan.allocate_output()
    g = torch.Generator(device=dev)
    g.manual_seed(1 + rank)
    u.data.uniform_(-1.0, 1.0, generator=g)
    stream = torch.cuda.current_stream()

    def step():
        P.mul_(v, plan, u)
        P.ldiv_(u, plan, v)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()

    def barrier():
        if world > 1:
            dist.barrier()

    # ---- timed region (device events on the launching stream) ----
    sampler = ClockSampler(local_rank)
    sampler.start()
    time.sleep(0.3)
    plan.set_timing(True)
    barrier()
    torch.cuda.synchronize()
    # one event between consecutive steps: the spread of the step times
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    evs[0].record(stream)
    for i in range(args.steps):
        step()
        evs[i + 1].record(stream)
    torch.cuda.synchronize()
    barrier()
    clocks = sampler.stop()
    ms_total = evs[0].elapsed_time(evs[-1])
    per_step = np.array([evs[i].elapsed_time(evs[i + 1]) for i in range(args.steps)])
    step_stats = {"mean": float(per_step.mean()), "std": float(per_step.std()),
                  "min": float(per_step.min()), "max": float(per_step.max()), "n": int(args.steps)}
    timing = plan.get_timing()
    plan.set_timing(False)
    ms_step = max_over_ranks(ms_total / args.steps, world, dev)

    # ---- roofline of the dominant kernel ----
    per_kernel = {}
    launches = 0
    for e in timing:
        k = per_kernel.setdefault(e["kernel"], {"ms": 0.0, "bytes": 0, "launches": 0})
        k["ms"] += e["total_ms"]
        k["bytes"] += e["bytes_per_launch"] * e["launches"]
        k["launches"] += e["launches"]
        launches += e["launches"]
    dom_name, dom = max(per_kernel.items(), key=lambda kv: kv[1]["ms"])
    avg_launch_s = dom["ms"] / dom["launches"] * 1e-3
    bytes_per_launch = dom["bytes"] / dom["launches"]
    achieved = bytes_per_launch / avg_launch_s / 1e9
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))
        peak, peak_src = float(peaks["hbm_gbs"]), "measured"
    except Exception:
        peak, peak_src = 6800.0, "fallback"
    traffic = None
    try:
        prof = json.load(open(os.path.join(REPO, "profiles", "traffic.json")))
        key = f"{dom_name}|{'x'.join(map(str, dims))}"
        if key in prof:
            traffic = prof[key]["dram_bytes_per_launch"]
    except Exception:
        pass
    alg_rt, R, C = alg_bytes_round_trip(dims, rb)

    # ---- end to end through the public API with host buffers ----
    # Every step copies its input from pinned host memory and its result back.
    # The copies run on their own streams, double-buffered, so the copy-in of
    # step k+1 and the copy-out of step k-1 overlap the transforms of step k.
    e2e = None
    if not args.no_e2e:
        host_in = torch.empty(u.data.shape, dtype=u.data.dtype, pin_memory=True)
        host_in.uniform_(-1.0, 1.0)
        host_out = [torch.empty_like(host_in, pin_memory=True) for _ in range(2)]
        us = [plan.allocate_input() for _ in range(2)]
        ws = [plan.allocate_input() for _ in range(2)]
        s_in, s_cmp, s_out = (torch.cuda.Stream(device=dev) for _ in range(3))
        ev_in = [torch.cuda.Event() for _ in range(2)]
        ev_cmp = [torch.cuda.Event() for _ in range(2)]
        ev_out = [torch.cuda.Event() for _ in range(2)]
        used = [False, False]

        def e2e_step(k):
            sl = k & 1
            if used[sl]:
                s_in.wait_event(ev_cmp[sl])    # transforms of step k-2 read us[sl]
                s_cmp.wait_event(ev_out[sl])   # copy-out of step k-2 read ws[sl]
            with torch.cuda.stream(s_in):
                us[sl].data.copy_(host_in, non_blocking=True)
                ev_in[sl].record(s_in)
            s_cmp.wait_event(ev_in[sl])
            with torch.cuda.stream(s_cmp):
                P.mul_(v, plan, us[sl])
                P.ldiv_(ws[sl], plan, v)
                ev_cmp[sl].record(s_cmp)
            s_out.wait_event(ev_cmp[sl])
            with torch.cuda.stream(s_out):
                host_out[sl].copy_(ws[sl].data, non_blocking=True)
                ev_out[sl].record(s_out)
            used[sl] = True

        for k in range(2):
            e2e_step(k)
        torch.cuda.synchronize()
        barrier()
        # three timed repetitions of the K steps, median reported: the host
        # link is shared with other jobs on the machine and varies run to run
        samples = []
        for _ in range(3):
            f0 = torch.cuda.Event(enable_timing=True)
            f1 = torch.cuda.Event(enable_timing=True)
            f0.record(s_in)
            for k in range(args.steps):
                e2e_step(k)
            s_in.wait_stream(s_out)
            f1.record(s_in)
            torch.cuda.synchronize()
            samples.append(f0.elapsed_time(f1) / args.steps)
        e2e_ms = max_over_ranks(statistics.median(samples), world, dev)
        nb = host_in.numel() * host_in.element_size()
        e2e = {"value": e2e_ms, "unit": UNIT, "h2d_bytes_per_step": nb, "d2h_bytes_per_step": nb,
               "pipelined": "copy-in / transforms / copy-out on three streams, double-buffered",
               "samples_ms": samples, "statistic": "median of 3 timed repetitions of the K steps"}
        # the result of the last step round-trips the input
        diff = host_out[(args.steps - 1) & 1].double() - host_in.double()
        e2e["round_trip_rel_l2"] = float(diff.norm() / host_in.double().norm())
        e2e["round_trip_max_rel"] = float(diff.abs().max() / host_in.double().abs().max())

    if rank != 0:
        return
    # cpu_baseline leg, as the checker: the GPU forward and ldiv! of the
    # benchmark's input against the oracle (scipy.fft, FP64, host threads)
    parity = None
    if not args.no_cpu_baseline:
        import scipy.fft as sfft
        from oracle import pencilfft_oracle as O
        x = u.to_logical()
        P.mul_(v, plan, u)
        got = v.to_logical()
        back = plan.ldiv(v).to_logical()
        orc = O.OraclePlan(dims, O.RFFT(), real)
        with sfft.set_workers(os.cpu_count() or 1):
            ref = orc.forward(x)
            e_fwd = _rel(got, ref)
            del ref
            e_bwd = _rel(back, orc.ldiv(got))
        parity = {"rel_l2_forward_vs_oracle": e_fwd, "rel_l2_backward_vs_oracle": e_bwd,
                  "rel_l2_round_trip": _rel(back, x),
                  "tolerance": 1e-13 if rb == 8 else 2e-6,
                  "oracle": "FP64 restatement of the reference path (scipy.fft), same input"}
        del x, got, back
    forms = None
    if not args.no_forms:
        forms = measure_forms(P, dims, args.steps, args.warmup, dev)
    del plan, u, v
    torch.cuda.empty_cache()
    configs = None
    if args.configs != "none":
        from oracle import pencilfft_oracle as O
        names = list(CONFIGS) if args.configs == "all" else args.configs.split(",")
        configs = {}
        for nm in names:
            try:
                configs[nm] = CONFIGS[nm](P, O, args.config_steps, 3)
            except Exception as e:  # a failing configuration is reported, not hidden
                configs[nm] = {"error": f"{type(e).__name__}: {e}"[:500]}
            torch.cuda.empty_cache()
    line = {
        "metric": METRIC, "value": ms_step, "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "step_ms": step_stats,
        "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if rb == 8 else "f32", "data": "synthetic: uniform [-1,1), seeded",
        "config": headline_config(args, world),
        "arithmetic": ARITHMETIC.get((args.real, args.precision), args.precision),
        # per direction: the forward (mul!) and backward (ldiv!) passes' device time
        "forward_ms": sum(e["total_ms"] for e in timing if e["direction"] > 0) / args.steps,
        "backward_ms": sum(e["total_ms"] for e in timing if e["direction"] < 0) / args.steps,
        "hbm_gbs": alg_rt / (ms_step * 1e-3) / 1e9 * world,
        # compulsory bytes: one read of the input and one write of the output
        # per direction, 2 (R + C)
        "compulsory_gbs": 2 * (R + C) / (ms_step * 1e-3) / 1e9 * world,
        "gflops": 2 * 2.5 * np.prod(dims) * np.log2(np.prod(dims)) / (ms_step * 1e-3) / 1e9 * world,
        "roofline": {"bound": "hbm", "kernel": dom_name, "achieved": achieved, "peak": peak,
                     "peak_source": peak_src, "unit": "GB/s", "frac": achieved / peak,
                     "traffic": traffic, "alg_bytes_per_launch": bytes_per_launch,
                     "avg_launch_ms": avg_launch_s * 1e3},
        "passes": [{k: e[k] for k in ("direction", "pass_", "axis", "launches", "total_ms",
                                      "bytes_per_launch", "kernel")} for e in timing],
        "cpu_baseline": cpu_baseline,
        "e2e": e2e,
        "gpu_launches": launches,
        "forms": forms,
        "clocks": clocks,
        "configs": configs,
    }
    if parity:
        line.update(parity)
    print(json.dumps(line), flush=True)


def run_reference(args, rank, world):
    """Reference arm: the CPU restatement of the path (oracle, scipy.fft on all
    host threads), the same workload and metric; rank 0 only."""
    if rank != 0:
        return
    dims, rb = workload(args)
    time_cpu_oracle(dims, rb, 0, max_iters=max(1, min(args.warmup, 1)))  # warm-up
    ms, iters, threads = time_cpu_oracle(dims, rb, 0, max_iters=args.steps)
    line = {
        "impl": "reference", "metric": METRIC, "value": ms, "unit": UNIT, "n_gpus": 0,
        "steps": iters, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64" if rb == 8 else "f32",
        "data": "synthetic: uniform [-1,1), seeded",
        "config": headline_config(args, world),
        "cpu_baseline": {"value": ms, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{iters} full round trips (oracle: scipy.fft pocketfft, "
                                   f"{threads} threads; Julia/FFTW are not installed)"},
        "e2e": {"value": ms, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def profile_batch():
    """The batch of configuration C5 (ii) in both forms, one launch each (the
    persistent launch first), for a kernel profiler."""
    import numpy as np
    import torch

    import pencilffts_gb300 as P
    T = P.Transforms
    rng = np.random.default_rng(2024)
    sizes = [tuple(int(s) for s in rng.integers(48, 193, 3)) for _ in range(64)]
    ops, keep = [], []
    for d in sizes:
        p = P.PencilFFTPlan(d, T.RFFT(), np.float32)
        u, v, w = p.allocate_input(), p.allocate_output(), p.allocate_input()
        u.copy_from_logical(rng.standard_normal(d).astype(np.float32))
        keep.append((p, u, v, w))
        ops += [(P.mul_, v, p, u), (P.ldiv_, w, p, v)]
    forms = [P.Batch(ops, form="persistent"), P.Batch(ops, form="graph")]
    for b in forms:
        b.launch()
    torch.cuda.synchronize()
    print(json.dumps({"profile_batch": [b.info() for b in forms]}))


def main():
    args = parse()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
        return
    if args.profile_batch:
        profile_batch()
        return
    if world > 1:
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl")
    try:
        run_gpu(args, rank, world, local_rank)
    finally:
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()


if __name__ == "__main__":
    main()
