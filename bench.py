#!/usr/bin/env python
"""Benchmark of the flagfft.h Exec hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload NAME | --problem TYPE:N:BATCH[:MODE]] [--no-extras]

Workloads (one step executes every call of the workload once):
  configs (default): the three plain-path configurations in one step --
      (1) C2C N = 4096 x 256, forward then inverse;
      (2) C2C N = 1701, 1009, 10007 x 1024 and Z2Z at the same lengths x 256,
          forward;
      (3) R2C -> C2R N = 2^24 x 4 (float), D2Z N = 3*2^20 x 2, 2-D C2C
          4096 x 4096, forward;
      all out of place.  The default run also measures (4) the batched
      uneven-length set and (5) the serving loop and carries them as the
      "batched_uneven" and "serving" keys of the same JSON line.
  arbitrary_1d, plain_c2c_4096, real_large: configuration 2, 1 or 3 alone.
  batched_uneven, serving: configuration 4 or 5 alone (its own JSON line).
Inputs are seeded uniform[-1, 1) (synthetic; no dataset).

Metric: GFLOP/s at 5 N log2 N per complex transform (2-D: 5 n0 n1 log2(n0 n1);
real transforms quoted at the same 5 N log2 N), whole job over all ranks.  The
JSON line also carries, per call, the device time, GFLOP/s and GB/s of
algorithmic bytes (P x batch x (N_in e_in + N_out e_out), P = 1 when one
transform fits on chip, else 2); per configuration the same totals and HBM
fraction; the roofline of the dominant kernel; the end-to-end figure through
the public API with host buffers; cuFFT (torch.fft) on the same calls; and
two CPU baselines on the host cores: the oracle port (the reference's
algorithms restated in C) on a bounded sample, and scipy.fft in FP64 on the
whole step.

Multi-GPU (torchrun): every rank runs the same per-GPU workload on its own GPU
(independent transforms: no collective on the data path, weak scaling); the
timing is the max over ranks.
"""
from __future__ import annotations

import argparse
import gc
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time
import traceback
from pathlib import Path

ROOT = Path(__file__).resolve().parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

from flagfft_b200.workloads import length_groups, serving_trace, uneven_lengths  # noqa: E402

# (type, N, batch, mode): mode "f" forward; "fi" forward then inverse back;
# "rt" R2C then C2R back.  Type "C2C2D" is an N x N 2-D C2C.
CONFIG1 = [("C2C", 4096, 256, "fi")]
CONFIG2 = [("C2C", 1701, 1024, "f"), ("C2C", 1009, 1024, "f"), ("C2C", 10007, 1024, "f"),
           ("Z2Z", 1701, 256, "f"), ("Z2Z", 1009, 256, "f"), ("Z2Z", 10007, 256, "f")]
CONFIG3 = [("R2C", 1 << 24, 4, "rt"), ("D2Z", 3 << 20, 2, "f"), ("C2C2D", 4096, 1, "f")]
WORKLOADS = {
    "configs": CONFIG1 + CONFIG2 + CONFIG3,
    "arbitrary_1d": CONFIG2,
    "plain_c2c_4096": CONFIG1,
    "real_large": CONFIG3,
    "batched_uneven": [],  # generated by uneven_lengths()
    "serving": [],  # generated by serving_trace()
    "precision": [],  # the precision-mode comparison (run_precision)
}
CONFIG_OF = {p: "1" for p in CONFIG1} | {p: "2" for p in CONFIG2} | {p: "3" for p in CONFIG3}
WORKLOAD_DESC = {
    "configs": "(1) C2C N=4096 x256 forward + inverse; (2) C2C N=1701,1009,10007 x1024 + Z2Z same N x256 forward; "
               "(3) R2C->C2R N=2^24 x4, D2Z N=3*2^20 x2, 2-D C2C 4096x4096 forward; all out-of-place",
    "arbitrary_1d": "C2C N=1701,1009,10007 x1024 + Z2Z same N x256, forward, out-of-place",
    "plain_c2c_4096": "C2C N=4096 x256, forward + inverse, out-of-place",
    "real_large": "R2C->C2R N=2^24 x4, D2Z N=3*2^20 x2, 2-D C2C 4096x4096, out-of-place",
    "batched_uneven": "10000 C2C transforms, lengths log-uniform in [16, 65536] (40% powers of two, 30% 7-smooth, "
                      "30% primes), forward, one batch plan (persistent launches + CUDA graph) vs the plain path",
    "serving": "Poisson arrivals at 50k req/s, requests C2C/R2C/Z2Z (60/30/10%), lengths as batched_uneven, "
               "batch 1-64, 40 GB HBM budget; request server (continuous batching) vs per-request Exec",
    "precision": "C2C N=4096 x8192 and N=256 x131072 forward: split-bf16 tcgen05 radix-16 stages (3 and 6 terms) "
                 "vs the plan path (SIMT codelets)",
}
TYPES = ("C2C", "Z2Z", "R2C", "D2Z", "C2R", "Z2D", "C2C2D")


def parse_args():
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=300)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--workload", choices=sorted(WORKLOADS), default="configs")
    ap.add_argument("--cpu-seconds", type=float, default=12.0, help="budget of the CPU baseline sample")
    ap.add_argument("--no-cufft", action="store_true")
    ap.add_argument("--no-extras", action="store_true",
                    help="skip the batched (config 4) and serving (config 5) keys of the default workload")
    ap.add_argument("--serve-seconds", type=float, default=10.0, help="arrival window of the serving workload")
    ap.add_argument("--serve-rate", type=float, default=50000.0, help="Poisson arrival rate (requests/s)")
    ap.add_argument("--problem", default=None, metavar="TYPE:N:BATCH[:MODE]",
                    help="run one problem instead of a named workload (profiling captures), e.g. C2C:10007:1024")
    args = ap.parse_args()
    if args.problem:
        parts = args.problem.split(":")
        t, n, b = parts[0], int(parts[1]), int(parts[2])
        mode = parts[3] if len(parts) > 3 else "f"
        if t not in TYPES or mode not in ("f", "fi", "rt") or (mode == "rt" and t not in ("R2C", "D2Z")):
            ap.error(f"bad problem {args.problem}")
        WORKLOADS["problem"] = [(t, n, b, mode)]
        WORKLOAD_DESC["problem"] = f"{t} N={n} x{b} mode {mode}, out-of-place"
        args.workload = "problem"
    return args


# ---------------------------------------------------------------------------
# helpers
# ---------------------------------------------------------------------------

def elem_bytes(t: str) -> tuple[int, int]:
    """(input element bytes, output element bytes)."""
    return {"C2C": (8, 8), "C2C2D": (8, 8), "Z2Z": (16, 16), "R2C": (4, 8), "D2Z": (8, 16), "C2R": (8, 4),
            "Z2D": (16, 8)}[t]


def flops_one(t: str, n: int, batch: int) -> float:
    """5 N log2 N per transform (real transforms quoted at the same figure;
    2-D N x N: 5 N^2 log2 N^2)."""
    if t == "C2C2D":
        return 5.0 * n * n * math.log2(n * n) * batch
    return 5.0 * n * math.log2(n) * batch


def calls_of(problem) -> list[tuple[str, int]]:
    """(type, direction) of each Exec call one step of the problem makes."""
    t, n, b, mode = problem
    if mode == "f":
        return [(t, -1)]
    if mode == "fi":
        return [(t, -1), (t, 1)]
    return [(t, -1), ({"R2C": "C2R", "D2Z": "Z2D"}[t], 1)]


def problem_flops(problem) -> float:
    t, n, b, mode = problem
    return flops_one(t, n, b) * len(calls_of(problem))


def max_over_ranks(values: list[float], device=None) -> list[float]:
    """Element-wise maximum of per-rank timings over the process group (the
    slowest rank times the job); the values themselves on one rank."""
    import torch
    import torch.distributed as dist
    if not (dist.is_available() and dist.is_initialized()) or dist.get_world_size() == 1:
        return list(values)
    t = torch.tensor(values, dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return t.tolist()


def job_value(step_flop: float, ms_step: float, world: int) -> float:
    """Whole-job GFLOP/s: every rank runs the same per-GPU step (replicas
    over batch), the step takes the slowest rank's time."""
    return step_flop * world / (ms_step * 1e-3) / 1e9


def measured_peaks() -> dict:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return {"hbm_gbs": float(d["hbm_gbs"]), "source": "measured (MEASURED_PEAKS.json hbm_gbs)"}
    return {"hbm_gbs": 6650.0, "source": "fallback 6.65 TB/s"}


def profiled_traffic() -> dict:
    """DRAM bytes per launch from committed ncu captures, keyed by call."""
    p = ROOT / "profiles" / "traffic.json"
    if not p.exists():
        return {}
    try:
        return json.loads(p.read_text())
    except ValueError:
        return {}


class ClockSampler:
    """SM clock / throttle-reason samples (NVML, read only, every ~2 ms) while
    the timed region runs; only samples taken inside the timed window are
    kept.  Falls back to `nvidia-smi -lms 50` when NVML is unavailable."""

    REASONS = {"hw_slowdown": 0x8, "hw_thermal_slowdown": 0x40, "sw_thermal_slowdown": 0x20, "sw_power_cap": 0x4}

    def __init__(self, device_index: int, pci_bus_id: str | None = None):
        self.dev = device_index
        self.pci = pci_bus_id
        self.samples: list[tuple[float, float, float, int]] = []  # (time, sm MHz, power W, reasons)
        self.sm_max = None
        self.stop_flag = threading.Event()
        self.thread = None
        self.proc = None
        self.window = (0.0, 0.0)

    def start(self):
        try:
            import pynvml
            pynvml.nvmlInit()
            h = (pynvml.nvmlDeviceGetHandleByPciBusId(self.pci) if self.pci
                 else pynvml.nvmlDeviceGetHandleByIndex(self.dev))
            self.sm_max = float(pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM))

            def poll():
                while not self.stop_flag.is_set():
                    try:
                        self.samples.append((time.time(), float(pynvml.nvmlDeviceGetClockInfo(h, pynvml.NVML_CLOCK_SM)),
                                             pynvml.nvmlDeviceGetPowerUsage(h) / 1000.0,
                                             int(pynvml.nvmlDeviceGetCurrentClocksEventReasons(h))))
                    except pynvml.NVMLError:
                        pass
                    time.sleep(0.002)

            self.thread = threading.Thread(target=poll, daemon=True)
            self.thread.start()
        except Exception:
            self._start_smi()
        time.sleep(0.1)

    def _start_smi(self):
        fields = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
                  "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
                  "clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.dev}", f"--query-gpu={fields}",
                                          "--format=csv,noheader,nounits", "-lms", "50"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except (OSError, FileNotFoundError):
            self.proc = None
            return

        def reader():
            bits = list(self.REASONS.values())
            for line in self.proc.stdout:
                parts = [p.strip() for p in line.split(",")]
                try:
                    r = sum(b for b, f in zip(bits, parts[3:7]) if f.lower() == "active")
                    self.sm_max = float(parts[1])
                    self.samples.append((time.time(), float(parts[0]), float(parts[2]), r))
                except (ValueError, IndexError):
                    continue

        self.thread = threading.Thread(target=reader, daemon=True)
        self.thread.start()

    def mark(self, t0: float, t1: float):
        self.window = (t0, t1)

    def stop(self) -> dict:
        self.stop_flag.set()
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
        if self.thread:
            self.thread.join(timeout=2)
        t0, t1 = self.window
        inside = [s for s in self.samples if t0 <= s[0] <= t1]
        where = "inside the timed window"
        if not inside:  # a window shorter than the sampling period: the samples nearest to it
            inside = [s for s in self.samples if t0 - 0.1 <= s[0] <= t1 + 0.1]
            where = "within 100 ms of a timed window shorter than the sampling period"
        if not inside:
            return {"sm_mhz": None, "sm_max_mhz": self.sm_max, "reasons": ["no samples near the timed window"]}
        reasons = sorted(name for name, bit in self.REASONS.items() if any(s[3] & bit for s in inside))
        return {"sm_mhz": statistics.median(s[1] for s in inside), "sm_max_mhz": self.sm_max, "reasons": reasons,
                "samples": len(inside), "power_w_max": max(s[2] for s in inside),
                "source": ("nvml" if self.proc is None else "nvidia-smi") + ", " + where}


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------

def executed_passes(description: str, direction: int) -> list[str]:
    """Pass lines of the program a call runs, from flagfftGetPlanDescription."""
    fwd = description.split("-- Forward execution --")[-1].split("-- Inverse execution --")[0]
    inv = description.split("-- Inverse execution --")[1] if "-- Inverse execution --" in description else fwd
    part = inv if direction > 0 else fwd
    return [ln.split(": ", 1)[1].strip() for ln in part.splitlines() if ln.strip().startswith("pass ")]


L2_BYTES = 126 * 2 ** 20


def step_footprint(problems) -> int:
    """Device bytes one step's calls read and write (distinct buffers)."""
    tot = 0
    for t0, n, b, mode in problems:
        for i, (t, _) in enumerate(calls_of((t0, n, b, mode))):
            ib, ob = elem_bytes(t)
            in_n = n // 2 + 1 if t in ("C2R", "Z2D") else n
            out_n = n // 2 + 1 if t in ("R2C", "D2Z") else n
            rows = n if t == "C2C2D" else b
            tot += (rows * in_n * ib if i == 0 else 0) + rows * out_n * ob
    return tot


def rotation_copies(problems) -> int:
    """Buffer sets a repeated call (or step) rotates through so that the
    bytes it touches between two uses of one set exceed twice the 126 MB L2:
    1 when one pass over them already does (at most 32 sets)."""
    return max(1, min(32, -(-2 * L2_BYTES // max(1, step_footprint(problems)))))


def build_calls(problems, dev, rank, torch, ffb):
    """Plans and device buffers of every Exec call of one step.  Each problem
    holds rotation_copies([problem]) buffer sets (`xs` / `ys`; a call's input
    set i is the previous call's output set i), so timing one call over and
    over never serves it from L2; `x` / `y` are set 0."""
    cdt = {"C2C": torch.complex64, "C2C2D": torch.complex64, "Z2Z": torch.complex128, "R2C": torch.float32,
           "D2Z": torch.float64, "C2R": torch.complex64, "Z2D": torch.complex128}
    odt = {"C2C": torch.complex64, "C2C2D": torch.complex64, "Z2Z": torch.complex128, "R2C": torch.complex64,
           "D2Z": torch.complex128, "C2R": torch.float32, "Z2D": torch.float64}
    tcode = {"C2C": ffb.C2C, "C2C2D": ffb.C2C, "Z2Z": ffb.Z2Z, "R2C": ffb.R2C, "D2Z": ffb.D2Z, "C2R": ffb.C2R,
             "Z2D": ffb.Z2D}
    gen = torch.Generator(device=dev)
    gen.manual_seed(0x46544646 + rank)

    def rand(shape, dt):
        if dt.is_complex:
            real = torch.float32 if dt == torch.complex64 else torch.float64
            return torch.view_as_complex((torch.rand((*shape, 2), generator=gen, device=dev, dtype=real) * 2 - 1)
                                         .contiguous())
        return torch.rand(shape, generator=gen, device=dev, dtype=dt) * 2 - 1

    calls = []
    for prob in problems:
        t0, n, b, mode = prob
        copies = rotation_copies([prob])
        src_ys = None
        for i, (t, direction) in enumerate(calls_of(prob)):
            in_n = n // 2 + 1 if t in ("C2R", "Z2D") else n
            out_n = n // 2 + 1 if t in ("R2C", "D2Z") else n
            shape_in = (n, n) if t == "C2C2D" else (b, in_n)
            shape_out = (n, n) if t == "C2C2D" else (b, out_n)
            xs = [rand(shape_in, cdt[t]) for _ in range(copies)] if src_ys is None else src_ys
            ys = [torch.empty(shape_out, dtype=odt[t], device=dev) for _ in range(copies)]
            plan = ffb.plan2d(n, n, tcode[t]) if t == "C2C2D" else ffb.plan1d(n, tcode[t], b)
            launches = plan.launch_count(direction)
            ib, ob = elem_bytes(t)
            elems_in = n * n if t == "C2C2D" else b * in_n
            elems_out = n * n if t == "C2C2D" else b * out_n
            passes = executed_passes(plan.description(), direction)
            calls.append({"t": t, "n": n, "b": b, "dir": direction, "x": xs[0], "y": ys[0], "xs": xs, "ys": ys,
                          "copies": copies, "plan": plan, "passes": passes, "config": CONFIG_OF.get(prob),
                          "key": f"{t}:{n}:{b}:{'fwd' if direction < 0 else 'inv'}",
                          "first": i == 0, "launches": launches,
                          "flop": flops_one(t, n, b),
                          "alg_bytes": (1 if launches == 1 else 2) * (elems_in * ib + elems_out * ob)})
            src_ys = ys
    return calls


def run_ours(args, rank: int, world: int, local_rank: int):
    import torch

    import flagfft_b200 as ffb

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    stream = torch.cuda.Stream(device=dev)
    calls = build_calls(WORKLOADS[args.workload], dev, rank, torch, ffb)
    for c in calls:
        c["plan"].set_stream(stream)
    it = [0]

    def step():
        i = it[0]
        it[0] += 1
        for c in calls:
            k = i % c["copies"]
            c["plan"].execute(c["xs"][k], c["ys"][k], c["dir"])

    # correctness spot check against cuFFT (torch.fft, FP64) on the first call, untimed
    check = None
    c0 = calls[0]
    if c0["t"] in ("C2C", "Z2Z"):
        with torch.cuda.stream(stream):
            c0["plan"].execute(c0["x"], c0["y"], c0["dir"])
        stream.synchronize()
        ref = torch.fft.fft(c0["x"].to(torch.complex128), dim=-1)
        err = (torch.linalg.vector_norm(c0["y"].to(torch.complex128) - ref, dim=-1) /
               torch.linalg.vector_norm(ref, dim=-1)).max().item()
        check = {"problem": c0["key"], "max_rel_l2_vs_cufft_fp64": err}

    def barrier():
        if world > 1:
            import torch.distributed as dist
            dist.barrier()

    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            step()
    torch.cuda.synchronize()

    # ---- whole-step timing
    props = torch.cuda.get_device_properties(dev)
    pci = None
    if all(hasattr(props, f) for f in ("pci_domain_id", "pci_bus_id", "pci_device_id")):
        pci = f"{props.pci_domain_id:08X}:{props.pci_bus_id:02X}:{props.pci_device_id:02X}.0"
    sampler = ClockSampler(torch.cuda.current_device(), pci)
    sampler.start()
    barrier()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    w0 = time.time()
    e0.record(stream)
    with torch.cuda.stream(stream):
        for _ in range(args.steps):
            step()
    e1.record(stream)
    torch.cuda.synchronize()
    w1 = time.time()
    barrier()
    sampler.mark(w0, w1)
    clocks = sampler.stop()
    total_ms = e0.elapsed_time(e1)

    # ---- per-call timing (same stream, events around repeated execs): the
    # headline rotates through the call's buffer sets, so every repeat reads
    # and writes HBM; "hot" repeats one set (served from L2 when a call's
    # buffers fit there)
    reps = max(5, min(args.steps, 50))

    def time_call(c, rotate):
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        ev[0].record(stream)
        with torch.cuda.stream(stream):
            for r in range(reps):
                k = r % c["copies"] if rotate else 0
                c["plan"].execute(c["xs"][k], c["ys"][k], c["dir"])
        ev[1].record(stream)
        torch.cuda.synchronize()
        return ev[0].elapsed_time(ev[1]) / reps

    def time_copy(c):
        """The same bytes moved by a device copy (input set -> output set,
        rotated like the call): the HBM floor of a one-pass call, launch
        included.  None when input and output differ in size."""
        if c["xs"][0].numel() * c["xs"][0].element_size() != c["ys"][0].numel() * c["ys"][0].element_size():
            return None
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        ev[0].record(stream)
        with torch.cuda.stream(stream):
            for r in range(reps):
                k = r % c["copies"]
                c["ys"][k].view(torch.uint8).copy_(c["xs"][k].view(torch.uint8))
        ev[1].record(stream)
        torch.cuda.synchronize()
        return ev[0].elapsed_time(ev[1]) / reps

    for c in calls:
        c["ms"] = time_call(c, True)
        c["ms_hot"] = time_call(c, False) if c["copies"] > 1 else c["ms"]
        c["copy_ms"] = time_copy(c)

    # ---- cuFFT comparator (torch.fft, same calls, same stream)
    cufft = None
    if not args.no_cufft:
        cufft = {}
        for c in calls:
            t, n = c["t"], c["n"]
            fn = {"C2C": lambda x: torch.fft.fft(x, dim=-1) if c["dir"] < 0 else torch.fft.ifft(x, dim=-1),
                  "Z2Z": lambda x: torch.fft.fft(x, dim=-1) if c["dir"] < 0 else torch.fft.ifft(x, dim=-1),
                  "R2C": lambda x: torch.fft.rfft(x, dim=-1), "D2Z": lambda x: torch.fft.rfft(x, dim=-1),
                  "C2R": lambda x: torch.fft.irfft(x, n=n, dim=-1), "Z2D": lambda x: torch.fft.irfft(x, n=n, dim=-1),
                  "C2C2D": lambda x: torch.fft.fft2(x)}[t]
            with torch.cuda.stream(stream):
                for _ in range(3):
                    fn(c["x"])
                ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                torch.cuda.synchronize()
                ev[0].record(stream)
                for r in range(reps):
                    fn(c["xs"][r % c["copies"]])
                ev[1].record(stream)
            torch.cuda.synchronize()
            ms = ev[0].elapsed_time(ev[1]) / reps
            cufft[c["key"]] = {"ms": ms, "gflops": c["flop"] / ms / 1e6}

    # ---- end-to-end through the public API with host buffers
    e2e = run_e2e(args, calls, stream, torch)

    # ---- max over ranks
    total_ms, e2e["ms_per_step"] = max_over_ranks([total_ms, e2e["ms_per_step"]], dev)
    for c in calls:
        c["plan"].destroy()
    return {"total_ms": total_ms, "calls": calls, "clocks": clocks, "check": check, "cufft": cufft, "e2e": e2e}


def run_e2e(args, calls, stream, torch):
    """Same step through the public API with host buffers: per step each
    problem's input is copied from pinned host memory, its calls run, and its
    final result is read back into pinned host memory.  Copies in, compute and
    copies out run on three streams ordered per problem by events, so one
    problem's transfers overlap another's transforms (as a serving pipeline
    would); the timed region spans from before the first input copy to after
    the last output copy."""
    groups = []  # (first call index, last call index) per problem
    for i, c in enumerate(calls):
        if c["first"]:
            groups.append([i, i])
        groups[-1][1] = i
    hin = [torch.empty(calls[a]["x"].shape, dtype=calls[a]["x"].dtype, pin_memory=True) for a, _ in groups]
    for h, (a, _) in zip(hin, groups):
        h.copy_(calls[a]["x"].cpu())
    hout = [torch.empty(calls[b]["y"].shape, dtype=calls[b]["y"].dtype, pin_memory=True) for _, b in groups]
    h2d = sum(h.numel() * h.element_size() for h in hin)
    d2h = sum(h.numel() * h.element_size() for h in hout)
    s_in, s_out = torch.cuda.Stream(), torch.cuda.Stream()
    ev = lambda: torch.cuda.Event()  # noqa: E731
    in_ready = [ev() for _ in groups]
    done = [ev() for _ in groups]
    out_free = [ev() for _ in groups]
    first_step = [True]

    def step():
        for g, (a, b) in enumerate(groups):
            with torch.cuda.stream(s_in):
                if not first_step[0]:
                    s_in.wait_event(done[g])  # the previous step's transforms finished reading x
                calls[a]["x"].copy_(hin[g], non_blocking=True)
                in_ready[g].record(s_in)
            stream.wait_event(in_ready[g])
            if not first_step[0]:
                stream.wait_event(out_free[g])  # the previous step's read-back of y finished
            for c in calls[a:b + 1]:
                c["plan"].execute(c["x"], c["y"], c["dir"])
            done[g].record(stream)
            with torch.cuda.stream(s_out):
                s_out.wait_event(done[g])
                hout[g].copy_(calls[b]["y"], non_blocking=True)
                out_free[g].record(s_out)
        first_step[0] = False

    for _ in range(max(1, args.warmup // 2)):
        step()
    torch.cuda.synchronize()
    steps = max(3, min(args.steps // 4, 50))
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    s_in.wait_event(e0)
    for _ in range(steps):
        step()
    stream.wait_stream(s_out)
    e1.record(stream)
    torch.cuda.synchronize()
    return {"ms_per_step": e0.elapsed_time(e1) / steps, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
            "steps": steps, "overlap": "copies in / transforms / copies out on three streams"}


# ---------------------------------------------------------------------------
# batched uneven lengths (one batch plan vs the plain path)
# ---------------------------------------------------------------------------

def run_batched(args, rank: int, world: int, local_rank: int):
    import torch

    import flagfft_b200 as ffb

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    stream = torch.cuda.Stream(device=dev)
    lengths = uneven_lengths()
    groups: dict[int, int] = {}
    for n in lengths:
        groups[n] = groups.get(n, 0) + 1
    glen = sorted(groups)
    gcnt = [groups[n] for n in glen]
    total = sum(n * c for n, c in zip(glen, gcnt))
    flop = sum(5.0 * n * math.log2(n) * c for n, c in zip(glen, gcnt))
    alg_bytes = 0
    gen = torch.Generator(device=dev)
    gen.manual_seed(0x46544646 + rank)
    x = torch.view_as_complex((torch.rand((total, 2), generator=gen, device=dev) * 2 - 1).contiguous())
    y = torch.empty_like(x)

    t0 = time.perf_counter()
    bplan = ffb.plan_batch(glen, gcnt, ffb.C2C)
    plan_s = time.perf_counter() - t0
    bplan.set_stream(stream)
    launches = bplan.launch_count(-1)

    def timed(fn, steps):
        with torch.cuda.stream(stream):
            for _ in range(args.warmup):
                fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        with torch.cuda.stream(stream):
            for _ in range(steps):
                fn()
        e1.record(stream)
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / steps

    # batched: one Exec of the batch plan per step (graph replay)
    sampler = ClockSampler(torch.cuda.current_device())
    sampler.start()
    w0 = time.time()
    ms_batch = timed(lambda: bplan.execute(x, y, -1), args.steps)
    sampler.mark(w0, time.time())
    clocks = sampler.stop()

    # plain per-length: one plan1d(n, C2C, count) Exec per distinct length
    plans = []
    off = 0
    for n, c in zip(glen, gcnt):
        p = ffb.plan1d(n, ffb.C2C, c)
        p.set_stream(stream)
        plans.append((p, x[off:off + n * c], y[off:off + n * c], p.launch_count(-1)))
        alg_bytes += (1 if plans[-1][3] == 1 else 2) * n * c * 16
        off += n * c

    def per_length():
        for p, xi, yi, _ in plans:
            p.execute(xi, yi, -1)

    ms_len = timed(per_length, max(3, args.steps // 10))

    # plain per-request: one Exec per transform with a cached plan1d(n, C2C, 1)
    single = {}
    for n in glen:
        p = ffb.plan1d(n, ffb.C2C, 1)
        p.set_stream(stream)
        single[n] = p
    views = []
    off = 0
    for n, c in zip(glen, gcnt):
        for i in range(c):
            views.append((single[n], x[off + i * n:off + (i + 1) * n], y[off + i * n:off + (i + 1) * n]))
        off += n * c

    def per_request():
        for p, xi, yi in views:
            p.execute(xi, yi, -1)

    ms_req = timed(per_request, 3)
    # correctness spot check of the batch output against the per-length plans
    bplan.execute(x, y, -1)
    torch.cuda.synchronize()
    yb = y.clone()
    per_length()
    torch.cuda.synchronize()
    max_diff = ((yb - y).abs().max() / y.abs().max()).item()

    for p, *_ in plans:
        p.destroy()
    for p in single.values():
        p.destroy()
    bplan.destroy()
    ms_batch, ms_len, ms_req = max_over_ranks([ms_batch, ms_len, ms_req], dev)
    n_tr = len(lengths)
    peaks = measured_peaks()
    gbs = alg_bytes / (ms_batch * 1e-3) / 1e9
    return {
        "metric": "transforms_per_s", "value": n_tr * world / (ms_batch * 1e-3), "unit": "transforms/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_batch,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "c64",
        "data": "synthetic (seeded uniform[-1,1) re/im; seeded length draw)",
        "config": {"workload": "batched_uneven", "problems": WORKLOAD_DESC["batched_uneven"],
                   "transforms": n_tr, "distinct_lengths": len(glen), "elements": total,
                   "l2": f"{2 * total * 8 / 1e9:.2f} GB in + out per step, above the 126 MB L2",
                   "parallelism": f"replicas, {world} GPU"},
        "gflops": flop * world / (ms_batch * 1e-3) / 1e9,
        "plain_per_length": {"ms": ms_len, "transforms_per_s": n_tr / (ms_len * 1e-3), "launches": sum(p[3] for p in plans)},
        "plain_per_request": {"ms": ms_req, "transforms_per_s": n_tr / (ms_req * 1e-3)},
        "speedup_vs_per_request": ms_req / ms_batch, "speedup_vs_per_length": ms_len / ms_batch,
        "roofline": {"bound": "hbm", "kernel": "batch phases (all launches of one Exec)", "achieved": gbs,
                     "peak": peaks["hbm_gbs"], "unit": "GB/s", "frac": gbs / peaks["hbm_gbs"], "traffic": None,
                     "peak_source": peaks["source"]},
        "gpu_launches": launches * args.steps, "plan_seconds": plan_s, "clocks": clocks,
        "check": {"max_rel_diff_batch_vs_per_length": max_diff},
    }


# ---------------------------------------------------------------------------
# serving: Poisson arrivals into the request server vs per-request Exec
# ---------------------------------------------------------------------------

def run_serving(args, rank: int, world: int, local_rank: int):
    import numpy as np
    import torch

    import flagfft_b200 as ffb

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    trace = serving_trace(args.serve_rate, args.serve_seconds, seed=0x5E4E + rank)
    code = {"C2C": ffb.C2C, "R2C": ffb.R2C, "Z2Z": ffb.Z2Z}
    # inputs: one read-only pool per type (every request reads from its start);
    # outputs: a circular arena, each request its own region
    maxb = 64 * 65536
    pools = {"C2C": torch.randn(maxb, dtype=torch.complex64, device=dev),
             "R2C": torch.randn(maxb, dtype=torch.float32, device=dev),
             "Z2Z": torch.randn(maxb, dtype=torch.complex128, device=dev)}
    arena = torch.empty(8 << 30, dtype=torch.uint8, device=dev)
    arena_ptr, arena_len = arena.data_ptr(), arena.numel()
    out_bytes = {"C2C": lambda n: 8 * n, "R2C": lambda n: 8 * (n // 2 + 1), "Z2Z": lambda n: 16 * n}

    def out_slots():
        pos = 0
        for t, ty, n, b in trace:
            need = (out_bytes[ty](n) * b + 255) // 256 * 256
            if pos + need > arena_len:
                pos = 0
            yield arena_ptr + pos
            pos += need

    srv = ffb.Server(hbm_budget_bytes=40 << 30, max_ticks=4)
    t0 = time.perf_counter()
    for ty, n in sorted({(ty, n) for _, ty, n, _ in trace}):
        srv.prepare(code[ty], n, -1)
    prep_s = time.perf_counter() - t0
    # warm up every kernel shape once
    for (t, ty, n, b), o in zip(trace[:200], out_slots()):
        srv.wait(srv.submit(code[ty], n, b, pools[ty].data_ptr(), o, -1))

    torch.cuda.synchronize()
    tickets, sub_t = [], []
    # (the collector's full passes over this loop's half-million objects
    # paused the submitting thread for up to ~100 ms, then released a burst)
    gc.collect()
    gc.disable()
    start = time.perf_counter()
    try:
        for (t, ty, n, b), o in zip(trace, out_slots()):
            while time.perf_counter() - start < t:
                pass
            tickets.append(srv.submit(code[ty], n, b, pools[ty].data_ptr(), o, -1))
            sub_t.append(time.perf_counter() - start)
    finally:
        gc.enable()
    submit_end = time.perf_counter() - start
    lat = np.array([srv.wait(tk) for tk in tickets])
    # the last completion (submit + the server's latency), not the end of
    # this Python loop over half a million tickets
    makespan = float(np.max(np.array(sub_t) + lat * 1e-3))
    stats = srv.stats()
    srv.close()
    transforms = sum(b for _, _, _, b in trace)

    # plain path on the same arrivals: each request is b Execs of a cached
    # plan1d(n, type, 1) issued when it arrives, on one stream; its latency
    # runs from its arrival to the event after its last Exec
    window = min(args.serve_seconds, 0.25)
    sub = [r for r in trace if r[0] < window]
    plans = {}
    for _, ty, n, _ in sub:
        if (ty, n) not in plans:
            plans[(ty, n)] = ffb.plan1d(n, code[ty], 1)
    stream = torch.cuda.Stream(device=dev)
    for p in plans.values():
        p.set_stream(stream)
    elem_in = {"C2C": 8, "R2C": 4, "Z2Z": 16}
    events = []
    torch.cuda.synchronize()
    base = torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(stream):
        base.record(stream)
        pstart = time.perf_counter()
        for (t, ty, n, b), o in zip(sub, out_slots()):
            while time.perf_counter() - pstart < t:
                pass
            p = plans[(ty, n)]
            ob = out_bytes[ty](n)
            for i in range(b):
                p.execute(pools[ty].data_ptr() + i * n * elem_in[ty], o + i * ob, -1)
            ev = torch.cuda.Event(enable_timing=True)
            ev.record(stream)
            events.append((t, ev))
    torch.cuda.synchronize()
    plain_lat = np.array([base.elapsed_time(ev) - t * 1e3 for t, ev in events])
    plain_makespan_ms = base.elapsed_time(events[-1][1])
    plain_transforms = sum(b for _, _, _, b in sub)
    for p in plans.values():
        p.destroy()
    return {
        "metric": "transforms_per_s", "value": transforms * world / makespan, "unit": "transforms/s",
        "n_gpus": world, "steps": 1, "warmup": 1, "ms_per_step": makespan * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "c64+f32+c128",
        "data": "synthetic (seeded Poisson trace; seeded uniform / normal inputs)",
        "config": {"workload": "serving", "problems": WORKLOAD_DESC["serving"], "requests": len(trace),
                   "transforms": transforms, "rate_req_s": args.serve_rate, "window_s": args.serve_seconds,
                   "l2": "outputs rotate through an 8 GB arena", "parallelism": f"replicas, {world} GPU"},
        "latency_ms": {"p50": float(np.percentile(lat, 50)), "p99": float(np.percentile(lat, 99)),
                       "mean": float(lat.mean())},
        "latency_p99_by_second_ms": [float(np.percentile(lat[(np.array(sub_t) >= k) & (np.array(sub_t) < k + 1)], 99))
                                     if np.any((np.array(sub_t) >= k) & (np.array(sub_t) < k + 1)) else None
                                     for k in range(int(math.ceil(args.serve_seconds)))],
        "offered_req_s": len(trace) / max(submit_end, 1e-9), "served_req_s": len(trace) / makespan,
        "ticks": stats["ticks"], "prepare_seconds": prep_s,
        "plain_per_request": {"window_s": window, "requests": len(sub),
                              "transforms_per_s": plain_transforms / (plain_makespan_ms * 1e-3),
                              "latency_ms": {"p50": float(np.percentile(plain_lat, 50)),
                                             "p99": float(np.percentile(plain_lat, 99))}},
        "speedup_vs_per_request": (transforms / makespan) / (plain_transforms / (plain_makespan_ms * 1e-3)),
    }


def precision_wait_failures(ffb) -> int:
    """The precision-mode kernel's count of bounded waits that gave up."""
    import ctypes
    v = ctypes.c_longlong(0)
    fn = ffb.LIB.flagfftB200PrecisionWaitFailures
    fn.argtypes = [ctypes.POINTER(ctypes.c_longlong)]
    fn.restype = ctypes.c_int
    return int(v.value) if fn(ctypes.byref(v)) == 0 else -1


def run_precision(args, rank: int, world: int, local_rank: int) -> dict:
    """Precision mode against the plan path on the same inputs: device time
    per call (inputs above the L2, CUDA events), GFLOP/s, and relative L2
    error of each against cuFFT in FP64 (torch.fft on complex128) over the
    first 64 transforms."""
    import ctypes

    import torch

    import flagfft_b200 as ffb
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    fn = ffb.LIB.flagfftB200PrecisionC2C
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                   ctypes.c_void_p]
    stream = torch.cuda.Stream(device=dev)
    out = {}
    for n, b in ((4096, 8192), (256, 131072)):
        g = torch.Generator(device=dev).manual_seed(n)
        x = torch.view_as_complex((torch.rand((b, n, 2), generator=g, device=dev) * 2 - 1).contiguous())
        y = torch.empty_like(x)
        ref = torch.fft.fft(x[:64].to(torch.complex128), dim=-1)
        plan = ffb.plan1d(n, ffb.C2C, b)
        plan.set_stream(stream)
        variants = {"plan_path": lambda: plan.execute(x, y, ffb.FORWARD)}
        for terms in (3, 6):
            variants[f"tensor_{terms}_terms"] = (lambda t=terms: fn(ctypes.c_void_p(x.data_ptr()),
                                                                   ctypes.c_void_p(y.data_ptr()), n, b, -1, t,
                                                                   ctypes.c_void_p(stream.cuda_stream)))
        res = {}
        for name, call in variants.items():
            fails0 = precision_wait_failures(ffb)
            reps = 20
            with torch.cuda.stream(stream):
                for _ in range(3):
                    call()
                ev = [torch.cuda.Event(enable_timing=True) for _ in range(reps + 1)]
                ev[0].record(stream)
                for r in range(reps):
                    call()
                    ev[r + 1].record(stream)
            torch.cuda.synchronize()
            per = sorted(ev[r].elapsed_time(ev[r + 1]) for r in range(reps))
            ms = statistics.median(per)
            err = (torch.linalg.vector_norm(y[:64].to(torch.complex128) - ref, dim=-1) /
                   torch.linalg.vector_norm(ref, dim=-1)).max().item()
            res[name] = {"ms": ms, "ms_min": per[0], "ms_max": per[-1],
                         "gflops": 5.0 * n * math.log2(n) * b / ms / 1e6,
                         "alg_GBs": 2 * 8 * n * b / ms / 1e6, "rel_l2_vs_fp64": err,
                         "bound": 5e-7 * math.log2(n),
                         "wait_failures": precision_wait_failures(ffb) - fails0}
        plan.destroy()
        out[f"C2C:{n}:{b}"] = res
    return out


# ---------------------------------------------------------------------------
# CPU baseline / reference arm: the oracle port of the reference algorithm
# ---------------------------------------------------------------------------

CPU_SAMPLE_DIV = 16  # the CPU port's sample of a problem: 1/16 of its rows (at least one transform)


def cpu_sample_rows(problem) -> int:
    t, n, b, mode = problem
    return max(1, b // CPU_SAMPLE_DIV)


def _cpu_inputs(problem, rows: int):
    """Seeded inputs of `rows` rows of a problem (uniform[-1, 1))."""
    import numpy as np
    from oracle import oracle as O
    t, n, b, mode = problem
    double = t in ("Z2Z", "D2Z")
    seed = O.accuracy_seed(O.C2C, n, rows)
    if t == "C2C2D":
        return O.random_complex(n * n, seed).reshape(1, n, n)
    if t in ("C2C", "Z2Z"):
        return O.random_complex(n * rows, seed, double).reshape(rows, n)
    return O.random_real(n * rows, seed, double).reshape(rows, n)


def port_problem(problem, x) -> tuple[float, float]:
    """Runs every call of `problem` on the rows of x with the oracle port --
    the reference's Exec algorithms restated in C (oracle/ffo.c), float
    arithmetic for single-precision types, double for double, on all host
    threads -- and returns (seconds, flop at 5 N log2 N)."""
    from oracle import oracle as O
    t, n, b, mode = problem
    prec = "f64" if t in ("Z2Z", "D2Z") else "f32"
    plans = O.ref_plans()
    tree = plans.get(f"{n}:{'z' if prec == 'f64' else 'c'}") or O.default_plan(n)
    rows = x.shape[0]
    t0 = time.perf_counter()
    if t == "C2C2D":
        O.fft2(x, "c2c", -1, row_plan=tree, col_plan=tree, precision=prec)
        flop = flops_one(t, n, 1)
    elif t in ("C2C", "Z2Z"):
        y = O.c2c(x, -1, tree, precision=prec)
        flop = flops_one(t, n, rows)
        if mode == "fi":
            O.c2c(y, 1, tree, precision=prec)
            flop *= 2
    else:
        y = O.r2c(x, tree, precision=prec)
        flop = flops_one(t, n, rows)
        if mode == "rt":
            O.c2r(y, n, tree, precision=prec)
            flop *= 2
    return time.perf_counter() - t0, flop


def scipy_problem(problem, x, workers: int) -> tuple[float, float]:
    """The same calls with scipy.fft in FP64 (pocketfft) on `workers` threads."""
    import numpy as np
    import scipy.fft as F
    t, n, b, mode = problem
    rows = x.shape[0]
    t0 = time.perf_counter()
    if t == "C2C2D":
        F.fft2(x, workers=workers)
        flop = flops_one(t, n, 1)
    elif t in ("C2C", "Z2Z"):
        y = F.fft(x, axis=-1, workers=workers)
        flop = flops_one(t, n, rows)
        if mode == "fi":
            F.ifft(y, axis=-1, norm="forward", workers=workers)
            flop *= 2
    else:
        y = F.rfft(x, axis=-1, workers=workers)
        flop = flops_one(t, n, rows)
        if mode == "rt":
            F.irfft(y, n=n, axis=-1, norm="forward", workers=workers)
            flop *= 2
    return time.perf_counter() - t0, flop


def cpu_baseline(problems, budget_s: float, threads: int) -> dict:
    """The oracle port on a bounded sample of the step: 1/16 of each
    problem's rows (at least one transform), every problem in turn, rounds
    until about budget_s seconds (at least one round)."""
    import numpy as np
    os.environ.setdefault("FFO_THREADS", str(threads))
    from oracle import oracle as O
    O.build()
    inputs = []
    for prob in problems:
        x = _cpu_inputs(prob, cpu_sample_rows(prob))
        if prob[0] in ("C2C", "R2C", "C2C2D"):
            x = x.astype(np.complex64 if np.iscomplexobj(x) else np.float32)
        inputs.append(x)
    sec = flop = 0.0
    rounds = 0
    t0 = time.perf_counter()
    while rounds == 0 or time.perf_counter() - t0 < budget_s:
        for prob, x in zip(problems, inputs):
            s_, f_ = port_problem(prob, x)
            sec += s_
            flop += f_
        rounds += 1
    return {"value": flop / sec / 1e9, "unit": "GFLOP/s", "cores": threads, "kind": "port",
            "sample": f"{rounds} round(s) over every problem of the step at 1/{CPU_SAMPLE_DIV} of its rows (at least "
                      f"one transform; the 2-D transform whole): the oracle port (the reference's Exec algorithms "
                      f"restated in C: float arithmetic for single precision, double for Z2Z/D2Z) on {threads} host "
                      f"threads, {sec:.1f}s of CPU work"}


def cpu_baseline_fp64(problems, budget_s: float, threads: int) -> dict:
    """scipy.fft (pocketfft) in FP64 on the whole step with `threads` workers."""
    import numpy as np
    inputs = [_cpu_inputs(p, 1 if p[0] == "C2C2D" else p[2]) for p in problems]
    sec = flop = 0.0
    steps = 0
    t0 = time.perf_counter()
    while steps == 0 or time.perf_counter() - t0 < budget_s:
        for prob, x in zip(problems, inputs):
            s_, f_ = scipy_problem(prob, x.astype(np.complex128 if np.iscomplexobj(x) else np.float64), threads)
            sec += s_
            flop += f_
        steps += 1
    return {"value": flop / sec / 1e9, "unit": "GFLOP/s", "cores": threads, "kind": "scipy.fft FP64",
            "sample": f"{steps} whole step(s) of the workload with scipy.fft (pocketfft) in FP64, workers={threads}, "
                      f"{sec:.1f}s"}


def run_reference(args, rank: int, world: int):
    """Reference arm: the reference's own Exec cannot run (see the note), so
    its CPU restatement (the oracle port) runs on the host cores.  A step is a
    bounded sample of the workload: one problem's calls on 1/16 of its rows
    (at least one transform), the problems taken in turn; W untimed steps,
    then K timed ones.  value = flop of the timed steps / their time."""
    if rank != 0:
        return 0
    import numpy as np
    problems = WORKLOADS[args.workload]
    if not problems:
        print(json.dumps({"impl": "reference", "unavailable": f"workload {args.workload} has no CPU restatement arm"}))
        return 0
    threads = os.cpu_count() or 1
    os.environ.setdefault("FFO_THREADS", str(threads))
    from oracle import oracle as O
    O.build()
    inputs = []
    for prob in problems:
        x = _cpu_inputs(prob, cpu_sample_rows(prob))
        if prob[0] in ("C2C", "R2C", "C2C2D"):
            x = x.astype(np.complex64 if np.iscomplexobj(x) else np.float32)
        inputs.append(x)
    per = {}
    step_ms = []
    sec = flop = 0.0
    for i in range(args.warmup + args.steps):
        k = i % len(problems)
        s_, f_ = port_problem(problems[k], inputs[k])
        if i >= args.warmup:
            sec += s_
            flop += f_
            step_ms.append(s_ * 1e3)
            key = "{}:{}:{}:{}".format(*problems[k])
            d = per.setdefault(key, {"seconds": 0.0, "flop": 0.0, "rows": inputs[k].shape[0]})
            d["seconds"] += s_
            d["flop"] += f_
    v = flop / sec / 1e9
    for d in per.values():
        d["gflops"] = d["flop"] / d["seconds"] / 1e9
    sample = (f"step i = problem i mod {len(problems)} of the workload on 1/{CPU_SAMPLE_DIV} of its rows (at least one "
              f"transform; the 2-D transform whole), oracle port (the reference's Exec algorithms restated in C: float "
              f"for single precision, double for Z2Z/D2Z) on {threads} host threads")
    line = {
        "impl": "reference", "metric": "gflops_5nlog2n", "value": v, "unit": "GFLOP/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": statistics.mean(step_ms),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": dtype_of(problems),
        "data": "synthetic (seeded uniform[-1,1))",
        "config": {"workload": args.workload, "problems": WORKLOAD_DESC[args.workload],
                   "step": "bounded sample: one problem per step, problems in turn"},
        "cpu_baseline": {"value": v, "unit": "GFLOP/s", "cores": threads, "kind": "port", "sample": sample},
        "e2e": {"value": v, "unit": "GFLOP/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "per_problem": per,
        "note": "reference arm = the oracle's CPU port of the reference's Exec algorithms on the host cores "
                "(the reference's own Triton-JIT Exec cannot be built: its libtriton_jit submodule and "
                "Triton TLE extension are absent)",
    }
    print(json.dumps(line))
    return 0


def dtype_of(problems) -> str:
    names = {"C2C": "c64", "C2C2D": "c64", "Z2Z": "c128", "R2C": "f32", "D2Z": "f64"}
    return "+".join(sorted({names[p[0]] for p in problems}))


# ---------------------------------------------------------------------------

def main():
    args = parse_args()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)

    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local_rank))
    if args.workload == "precision":
        res = run_precision(args, rank, world, local_rank)
        if rank == 0:
            print(json.dumps({"metric": "precision_mode_comparison", "config": {"workload": "precision",
                              "problems": WORKLOAD_DESC["precision"]}, "results": res}))
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()
        return 0
    if args.workload in ("batched_uneven", "serving"):
        line = (run_batched if args.workload == "batched_uneven" else run_serving)(args, rank, world, local_rank)
        if rank == 0:
            print(json.dumps(line))
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()
        return 0
    res = run_ours(args, rank, world, local_rank)
    problems = WORKLOADS[args.workload]
    step_flop = sum(problem_flops(p) for p in problems)
    ms_step = res["total_ms"] / args.steps
    value = job_value(step_flop, ms_step, world)
    peaks = measured_peaks()
    traffic = profiled_traffic()

    per_call = []
    dominant = None
    for c in res["calls"]:
        gbs = c["alg_bytes"] / (c["ms"] * 1e-3) / 1e9
        row = {"call": c["key"], "config": c["config"], "passes": c["passes"], "ms": c["ms"],
               "gflops": c["flop"] / c["ms"] / 1e6, "alg_GBs": gbs, "hbm_frac": gbs / peaks["hbm_gbs"],
               "launches": c["launches"], "alg_bytes": c["alg_bytes"],
               "ms_per_launch": c["ms"] / max(1, c["launches"]), "ms_hot": c["ms_hot"],
               "rotation_sets": c["copies"], "copy_ms": c["copy_ms"]}
        per_call.append(row)
        if dominant is None or row["ms_per_launch"] > dominant["ms_per_launch"]:
            dominant = row
    launches_per_step = sum(c["launches"] for c in res["calls"])

    # per configuration: its calls' device time, GFLOP/s and algorithmic GB/s
    configs = {}
    for row, c in zip(per_call, res["calls"]):
        if not c["config"]:
            continue
        d = configs.setdefault(c["config"], {"calls": [], "ms": 0.0, "flop": 0.0, "alg_bytes": 0.0})
        d["calls"].append(row["call"])
        d["ms"] += row["ms"]
        d["flop"] += c["flop"]
        d["alg_bytes"] += row["alg_bytes"]
    for d in configs.values():
        d["gflops"] = d["flop"] / (d["ms"] * 1e-3) / 1e9
        d["alg_GBs"] = d["alg_bytes"] / (d["ms"] * 1e-3) / 1e9
        d["hbm_frac"] = d["alg_GBs"] / peaks["hbm_gbs"]
        if res["cufft"]:
            cms = sum(res["cufft"][k]["ms"] for k in d["calls"])
            d["cufft_ms"] = cms
            d["speedup_vs_cufft"] = cms / d["ms"]

    extras = {}
    if rank == 0 and world == 1 and args.workload == "configs" and not args.no_extras:
        extras["batched_uneven"] = _leg("batched_uneven", lambda: _extra(run_batched(args, rank, world, local_rank)))
        extras["serving"] = _leg("serving", lambda: _extra(serving_in_child(args)))
        extras["precision_mode"] = _leg("precision_mode", lambda: run_precision(args, rank, world, local_rank))

    if rank == 0:
        e2e_ms = res["e2e"]["ms_per_step"]
        alg_per_launch = dominant["alg_bytes"] / max(1, dominant["launches"])
        achieved = alg_per_launch / (dominant["ms_per_launch"] * 1e-3) / 1e9
        tr = traffic.get(dominant["call"])
        if tr and tr.get("passes") != dominant["passes"]:
            tr = None  # the capture was of another lowering of this call
        line = {
            "metric": "gflops_5nlog2n", "value": value, "unit": "GFLOP/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": dtype_of(problems),
            "data": "synthetic (seeded uniform[-1,1) re/im)",
            "config": {"workload": args.workload, "problems": WORKLOAD_DESC[args.workload],
                       "l2": (f"one step touches {step_footprint(problems) / 2 ** 20:.0f} MiB of distinct buffers"
                              + (", above the 126 MB L2; " if step_footprint(problems) > 2 * L2_BYTES else "; ")
                              + "each call's buffers rotate through enough sets that a buffer's next use comes "
                                "after more than twice the L2 of other traffic (per_call rotation_sets); "
                                "per_call ms_hot repeats one set"),
                       "parallelism": f"replicas over batch, {world} GPU"},
            "per_call": per_call,
            "configs": configs,
            "roofline": {"bound": "hbm", "kernel": dominant["call"], "passes": dominant["passes"],
                         "achieved": achieved, "peak": peaks["hbm_gbs"], "unit": "GB/s",
                         "frac": achieved / peaks["hbm_gbs"],
                         "traffic": tr["dram_bytes_per_launch"] if tr else None,
                         "traffic_source": tr["source"] if tr else None,
                         "peak_source": peaks["source"], "alg_bytes_per_launch": alg_per_launch,
                         "ms_per_launch": dominant["ms_per_launch"],
                         "dominant": "the call with the longest device time per launch",
                         # what bounds the kernel when HBM does not: the same capture's
                         # issue-slot, FMA-pipe and DRAM utilisation (duration-weighted)
                         "ncu_utilisation_pct": ({"issue_active": tr.get("issue_active_pct"),
                                                  "fma_pipe": tr.get("fma_pipe_pct"),
                                                  "dram_throughput": tr.get("dram_throughput_pct")} if tr else None)},
            "e2e": {"value": step_flop * world / (e2e_ms * 1e-3) / 1e9, "unit": "GFLOP/s",
                    "h2d_bytes_per_step": res["e2e"]["h2d_bytes_per_step"],
                    "d2h_bytes_per_step": res["e2e"]["d2h_bytes_per_step"], "ms_per_step": e2e_ms},
            "gpu_launches": launches_per_step * args.steps,
            "clocks": res["clocks"],
            "check": res["check"],
            "cufft": res["cufft"],
        }
        line.update(extras)
        if world == 1:
            threads = os.cpu_count() or 1
            line["cpu_baseline"] = cpu_baseline(problems, args.cpu_seconds, threads)
            line["cpu_baseline_fp64"] = cpu_baseline_fp64(problems, min(args.cpu_seconds, 5.0), threads)
        print(json.dumps(line))
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()
    return 0


def serving_in_child(args) -> dict:
    """The serving workload's line from a fresh process (this one has run
    the other workloads: their allocations and threads would share the
    window), as `python bench.py --workload serving` gives it."""
    cmd = [sys.executable, str(Path(__file__).resolve()), "--workload", "serving",
           "--serve-seconds", str(args.serve_seconds), "--serve-rate", str(args.serve_rate)]
    out = subprocess.run(cmd, stdout=subprocess.PIPE, text=True)  # (its messages go where this one's go)
    if out.returncode != 0:
        raise RuntimeError(f"the serving workload's process ended with status {out.returncode}")
    return json.loads(out.stdout.strip().splitlines()[-1])


def _leg(name: str, run) -> dict:
    """An extra key of the default line; one that fails is reported under its
    key and does not take the finished measurements with it."""
    try:
        return run()
    except Exception as e:  # noqa: BLE001
        traceback.print_exc()
        print(f"bench: the {name} leg failed: {e}", file=sys.stderr, flush=True)
        return {"error": f"{type(e).__name__}: {e}"}


def _extra(line: dict) -> dict:
    """A configuration-4 / -5 result as a key of the default line (its own
    metric, value, timing, comparisons and clocks)."""
    drop = {"n_gpus", "steps", "warmup", "higher_is_better", "scaling", "vs_baseline", "data"}
    return {k: v for k, v in line.items() if k not in drop}


if __name__ == "__main__":
    sys.exit(main())
