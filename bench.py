"""Benchmark: AMIPS + envelope queries/s on the isolated FP64 query batches.

Workload (one step): 4,000,000 tets from regular tets of edge 0.01 in the
unit cube, every vertex perturbed by N(0, 0.1 edge): orientation + AMIPS
energy (calTetQuality_AMIPS sentinel), gradient and Hessian; plus
10,000,000 points offset along the normal by U(-2 eps, 2 eps) around a
100,000-triangle displaced sphere, eps = 1e-3: squared distance <= eps^2.
A query is one tet E+J+H evaluation or one point-envelope decision, so a
step is 14,000,000 queries.  Inputs are seeded synthetic data of those
shapes (no dataset is available); all inputs exceed the 129 MB L2.

``value`` times the device-resident kernels (inputs already in HBM);
``e2e`` times the same step through the C-ABI with host buffers (pinned),
host<->device copies included.  ``--impl reference`` times the reference's
own CPU code (oracle/_ref) on a bounded sample with all host threads.

Multi-GPU: the queries are independent and every box has one GPU, so
``--gpus N`` under torchrun runs N replicas (weak scaling) with a barrier and
the max over ranks; there is no data-path collective.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

N_TETS = 4_000_000
N_POINTS = 10_000_000
EPS = 1e-3
GRID_CELL = 0.1   # envelope grid cell / mean facet extent (TW_TUNE_GRID_CELL)
METRIC = "AMIPS+envelope queries/s vs plain FP64 GPU at 0 decision mismatches; p99 ms"
UNIT = "queries/s"
BYTES_PER_TET = 96 + 8 + 24 + 72 + 1     # coords in; E, J, H, flip out
BYTES_PER_POINT = 24 + 1                 # point in; decision out
# The CPU legs time the whole step's work (about 1 us per query and thread
# on the host cores, so a few seconds with all threads).
CPU_SAMPLE_TETS = N_TETS
CPU_SAMPLE_POINTS = N_POINTS


def set_sizes(tets: int, points: int):
    """Profiling runs use a smaller case of the same workload; the benchmark line
    always uses the default sizes."""
    global N_TETS, N_POINTS, CPU_SAMPLE_TETS, CPU_SAMPLE_POINTS
    N_TETS, N_POINTS = tets, points
    CPU_SAMPLE_TETS, CPU_SAMPLE_POINTS = tets, points


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d.get("hbm_gbs", 6800.0)), "measured"
    return 6800.0, "fallback"


class NvmlClockSampler:
    """SM clock and clock-event (throttle) reasons read through NVML (the driver's
    libnvidia-ml, by ctypes) every 2 ms during the timed region: a timed region of
    tens of milliseconds still gets a record of several samples.  Reads only."""

    # nvmlClocksEventReasons bits
    REASONS = {0x4: "sw_power_cap", 0x8: "hw_slowdown", 0x20: "sw_thermal_slowdown",
               0x40: "hw_thermal_slowdown", 0x80: "hw_power_brake_slowdown"}
    PERIOD_S = 0.002

    def __init__(self, device: int, lib=None):
        import ctypes

        self.device = device
        self.samples = []   # (sm_mhz, reasons bitmask)
        self.sm_max = None
        self.ok = False
        self._stop = threading.Event()
        if device < 0:
            return
        try:
            L = lib or ctypes.CDLL("libnvidia-ml.so.1")
        except OSError:
            return
        self.L = L
        self.h = ctypes.c_void_p()
        if L.nvmlInit_v2() != 0:
            return
        if L.nvmlDeviceGetHandleByIndex_v2(ctypes.c_uint(device), ctypes.byref(self.h)) != 0:
            L.nvmlShutdown()
            return
        self._reasons = getattr(L, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
            getattr(L, "nvmlDeviceGetCurrentClocksThrottleReasons", None)
        mx = ctypes.c_uint()
        if L.nvmlDeviceGetMaxClockInfo(self.h, 1, ctypes.byref(mx)) == 0:   # NVML_CLOCK_SM
            self.sm_max = float(mx.value)
        self.ok = self._reasons is not None

    def _run(self):
        import ctypes

        clk, rs = ctypes.c_uint(), ctypes.c_ulonglong()
        while not self._stop.is_set():
            if (self.L.nvmlDeviceGetClockInfo(self.h, 1, ctypes.byref(clk)) == 0 and
                    self._reasons(self.h, ctypes.byref(rs)) == 0):
                self.samples.append((float(clk.value), int(rs.value)))
            time.sleep(self.PERIOD_S)

    def __enter__(self):
        if self.ok:
            self.t = threading.Thread(target=self._run, daemon=True)
            self.t.start()
        return self

    def __exit__(self, *a):
        if self.ok:
            self._stop.set()
            self.t.join(timeout=2)
            self.L.nvmlShutdown()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": self.sm_max, "reasons": [], "samples": 0,
                    "source": "nvml"}
        reasons = set()
        for _, r in self.samples:
            for bit, name in self.REASONS.items():
                if r & bit:
                    reasons.add(name)
        return {"sm_mhz": statistics.median(c for c, _ in self.samples),
                "sm_max_mhz": self.sm_max, "reasons": sorted(reasons),
                "samples": len(self.samples), "source": "nvml, every 2 ms"}


def clock_sampler(device: int):
    """NVML sampling when the driver library is loadable, else nvidia-smi."""
    s = NvmlClockSampler(device)
    return s if s.ok else ClockSampler(device)


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.lines = []

    def __enter__(self):
        if self.device < 0:
            return self
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except (FileNotFoundError, OSError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            self.t.join(timeout=2)

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in self.lines:
            parts = [x.strip() for x in l.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for name, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(name)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


def make_inputs(seed=0):
    from tetwild_gb300 import synthetic as syn

    T = syn.energy_batch(N_TETS, seed=seed)
    V, F = syn.displaced_sphere(seed=seed)
    P = syn.envelope_points(V, F, N_POINTS, EPS, seed=seed + 1)
    return T, V, F, P


def cpu_baseline(T, V, F, P, nthreads, frac=1):
    """The reference's own CPU code when oracle/_ref is built, else the oracle port,
    on a bounded sample (CPU_SAMPLE_TETS tets + CPU_SAMPLE_POINTS points, divided by
    frac)."""
    from oracle.oracle import Oracle, RefLib

    nt, npts = CPU_SAMPLE_TETS // frac, CPU_SAMPLE_POINTS // frac
    Ts = np.ascontiguousarray(T[:, :nt])
    Ps = np.ascontiguousarray(P[:npts])
    kind = "port"
    try:
        ref = RefLib()
        kind = "reference"
    except Exception:
        ref = None
    o = Oracle()
    if kind == "reference":
        S = ref.surface(V, F)
        t0 = time.perf_counter()
        ref.amips_batch_soa(Ts, nthreads=nthreads)
        o.amips_batch_soa(Ts, quality=True, nthreads=nthreads, jacobian=False, hessian=False)
        S.points_out(Ps, EPS * EPS, nthreads=nthreads)
        dt = time.perf_counter() - t0
        sample = (f"{nt} tets (reference comformalAMIPS E/J/H + oracle exact orientation) "
                  f"+ {npts} points (reference isPointOutEnvelop over MeshFacetsAABBWithEps)")
    else:
        S = o.surface(V, F)
        t0 = time.perf_counter()
        o.amips_batch_soa(Ts, quality=True, nthreads=nthreads)
        S.points_out(Ps, EPS * EPS, nthreads=nthreads)
        dt = time.perf_counter() - t0
        sample = f"{nt} tets E/J/H + {npts} points (oracle port)"
    q = nt + npts
    return {"value": q / dt, "unit": UNIT, "cores": nthreads, "kind": kind, "sample": sample,
            "seconds": dt}


def run_reference(args):
    ws, rank, _ = dist_env()
    if rank != 0:
        return 0
    from oracle.oracle import default_threads

    T, V, F, P = make_inputs()
    nthreads = default_threads()
    for _ in range(args.warmup):
        cpu_baseline(T, V, F, P, nthreads)
    times = []
    kind = sample = None
    for _ in range(args.steps):
        r = cpu_baseline(T, V, F, P, nthreads)
        times.append(r["seconds"])
        kind, sample = r["kind"], r["sample"]
    q = CPU_SAMPLE_TETS + CPU_SAMPLE_POINTS
    total = sum(times)
    value = q * args.steps / total
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic",
        "config": {"workload": "isolated query batches, FP64 plain: energy 4M tets E/J/H + envelope "
                               "10M points vs 100k-tri displaced sphere (bounded CPU sample per step)",
                   "sample_tets": CPU_SAMPLE_TETS, "sample_points": CPU_SAMPLE_POINTS},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": nthreads, "kind": kind,
                         "sample": sample},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def load_traffic():
    """Per-launch DRAM bytes of the dominant kernel from the committed ncu summary."""
    p = ROOT / "profiles" / "traffic.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except ValueError:
            return {}
    return {}


def run_ours(args):
    import torch

    import tetwild_gb300 as tw

    ws, rank, local = dist_env()
    if ws > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl" if torch.cuda.is_available() else "gloo")
    dev = local if ws > 1 else 0
    torch.cuda.set_device(dev)
    if args.only_batching:        # profiling runs of the star-batch pass alone (no line)
        from tetwild_gb300 import synthetic as syn

        V, F = syn.displaced_sphere(seed=rank)
        ctx = tw.Context(dev)
        ctx.set_params(EPS * EPS, EPS)
        ctx.surface_upload(V, F)
        r = run_batching(ctx, V, F, args, dev, ws)
        print(json.dumps({k: r[k] for k in ("stars", "tets", "value", "unit")}), flush=True)
        ctx.close()
        return 0
    T, V, F, P = make_inputs(seed=rank)
    ctx = tw.Context(dev)
    ctx.set_params(EPS * EPS, EPS)
    # a finer envelope grid than the default 0.2 (4% faster point tests through
    # the grid's hashed cells, the path of --bin-cell 0, for 4x the grid
    # memory); the default point test reads the bin index; results never
    # depend on either
    ctx.set_tuning(tw.Context.TUNE_GRID_CELL, GRID_CELL)
    if args.bin_cell is not None:
        ctx.set_tuning(tw.Context.TUNE_BIN_CELL, args.bin_cell)
    ctx.surface_upload(V, F)
    fp64_tflops, fp32_tflops = ctx.probe_peaks()

    stream = torch.cuda.ExternalStream(ctx.stream(), device=f"cuda:{dev}")
    d = torch.device(f"cuda:{dev}")
    dT = torch.from_numpy(T).to(d)
    dP = torch.from_numpy(P).to(d)
    dE = torch.empty(N_TETS, dtype=torch.float64, device=d)
    dJ = torch.empty(3 * N_TETS, dtype=torch.float64, device=d)
    dH = torch.empty(9 * N_TETS, dtype=torch.float64, device=d)
    dFl = torch.empty(N_TETS, dtype=torch.uint8, device=d)
    dO = torch.empty(N_POINTS, dtype=torch.uint8, device=d)
    torch.cuda.synchronize()

    def step(ev=None):
        if ev:
            ev[0].record(stream)
        ctx.amips_device(dT.data_ptr(), N_TETS, tw.TW_ENERGY_QUALITY, dE.data_ptr(), dJ.data_ptr(),
                         dH.data_ptr(), dFl.data_ptr())
        if ev:
            ev[1].record(stream)
        ctx.envelope_points_device(dP.data_ptr(), N_POINTS, dO.data_ptr())
        if ev:
            ev[2].record(stream)

    def measure(mode, clocks=True):
        """W warm-up steps, a correctness gate on this workload, then exactly K timed steps."""
        ctx.set_precision(mode)
        for _ in range(args.warmup):
            step()
        ctx.synchronize()
        mism = check_sample(T, P, V, F, dE, dFl, dO)
        ctx.reset_stats()
        evs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(args.steps)]
        ctx.set_tuning(ctx.TUNE_TIME_KERNELS, 1)   # events around the point-test kernel itself
        barrier(ws)
        torch.cuda.synchronize()
        with clock_sampler(dev if clocks else -1) as clk:
            t0 = time.perf_counter()
            for k in range(args.steps):
                step(evs[k])
            ctx.synchronize()
            torch.cuda.synchronize()
            wall = time.perf_counter() - t0
        t_kernel = ctx.kernel_times(64)
        ctx.set_tuning(ctx.TUNE_TIME_KERNELS, 0)
        t_amips = [evs[k][0].elapsed_time(evs[k][1]) for k in range(args.steps)]
        t_env = [evs[k][1].elapsed_time(evs[k][2]) for k in range(args.steps)]
        step_ms = [a + b for a, b in zip(t_amips, t_env)]
        dev_ms = max_over_ranks(sum(step_ms), ws)
        st = ctx.stats()
        return {"value": ws * (N_TETS + N_POINTS) * args.steps / (dev_ms * 1e-3),
                "ms_per_step": dev_ms / args.steps, "step_ms": step_ms,
                "t_amips": statistics.mean(t_amips), "t_env": statistics.mean(t_env),
                "t_env_kernel": statistics.mean(t_kernel) if t_kernel else None,
                "mism": mism, "stats": st, "clocks": clk.summary() if clocks else None,
                "wall": wall}

    modes = args.modes.split(",")
    cert = measure(tw.TW_PRECISION_FP32_CERTIFIED) if "cert" in modes else None
    plain = measure(tw.TW_PRECISION_FP64) if "plain" in modes else None
    if cert is None or plain is None:   # profiling runs: one mode, no benchmark line
        ctx.close()
        return 0
    ctx.set_precision(tw.TW_PRECISION_FP32_CERTIFIED)
    value = cert["value"]

    # e2e: the same step through the C-ABI with pinned host buffers, in both modes
    e2e = e2e_fp64 = None
    if not args.no_e2e:
        ctx.set_precision(tw.TW_PRECISION_FP64)
        e2e_fp64 = run_e2e(ctx, T, P, args, ws, steps=max(3, min(args.steps, 5)))
        ctx.set_precision(tw.TW_PRECISION_FP32_CERTIFIED)
        e2e = run_e2e(ctx, T, P, args, ws)

    hbm_peak, peak_kind = measured_peaks()
    ma, me = cert["t_amips"], cert["t_env"]
    mk = cert["t_env_kernel"] or me
    if mk >= ma:
        dom = {"kernel": "k_env_points_bins", "ms": mk, "bytes": BYTES_PER_POINT * N_POINTS,
               "units": N_POINTS, "per_unit": BYTES_PER_POINT}
    else:
        dom = {"kernel": "k_amips_soa_cert", "ms": ma, "bytes": BYTES_PER_TET * N_TETS,
               "units": N_TETS, "per_unit": BYTES_PER_TET}
    achieved = dom["bytes"] / (dom["ms"] * 1e-3) / 1e9
    traffic = load_traffic().get(dom["kernel"])
    traffic_bytes = None
    if traffic and traffic.get("bytes_per_unit"):
        traffic_bytes = traffic["bytes_per_unit"] * dom["units"]
    # the step's other kernel against the same peak (CUDA events around its launch)
    am_ach = BYTES_PER_TET * N_TETS / (ma * 1e-3) / 1e9
    am_tr = load_traffic().get("k_amips_soa_cert")
    roof_other = [{"kernel": "k_amips_soa_cert_bulk", "bound": "hbm", "achieved": am_ach,
                   "peak": hbm_peak, "unit": "GB/s", "frac": am_ach / hbm_peak,
                   "traffic": am_tr["bytes_per_unit"] * N_TETS if am_tr else None,
                   "algorithmic_bytes_per_unit": BYTES_PER_TET}]
    # FP64 instructions per tet of the plain kernel in the default (reference) energy
    # form: 466 distinct operations of E/J/H after common-subexpression elimination
    # (227 mul, 142 add, 90 sub, 4 div, 3 pow), ~20 per pow (icbrt's two binary64
    # Newton steps and the exponent correction) and ~30 for the orientation filter;
    # every one is a separate instruction (no FP contraction), so the pipe's peak is
    # half its FMA flop rate
    flops_per_tet = 556.0
    fp64_achieved = flops_per_tet * N_TETS / (plain["t_amips"] * 1e-3) / 1e12
    cst = cert["stats"]
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": cert["ms_per_step"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "fp32-certified+fp64-recheck",
        "data": "synthetic",
        "config": {"workload": "isolated query batches: energy 4M tets (orientation + AMIPS "
                               "E/J/H) + envelope 10M points vs a 100k-tri displaced sphere, "
                               "eps=1e-3; certified FP32 mode (decisions identical to FP64)",
                   "tets": N_TETS, "points": N_POINTS, "surface_tris": int(len(F)),
                   "l2": "inputs larger than L2 (384 MB tets, 240 MB points); no flush",
                   "grid_cell": GRID_CELL, "parallelism": f"replicas x{ws}"},
        "p50_ms": float(np.percentile(cert["step_ms"], 50)),
        "p99_ms": float(np.percentile(cert["step_ms"], 99)),
        "kernels_ms": {"amips_step": ma, "envelope_step": me,
                       "envelope_point_kernel": cert["t_env_kernel"]},
        "decision_mismatches": cert["mism"],
        "plain_fp64": {"dtype": "f64 (reference energy form)", "value": plain["value"],
                       "ms_per_step": plain["ms_per_step"],
                       "kernels_ms": {"amips_step": plain["t_amips"],
                                      "envelope_step": plain["t_env"],
                                      "envelope_point_kernel": plain["t_env_kernel"]},
                       "decision_mismatches": plain["mism"],
                       "p99_ms": float(np.percentile(plain["step_ms"], 99)),
                       "e2e": e2e_fp64,
                       "speedup_of_value": value / plain["value"],
                       "speedup_of_e2e": (e2e["value"] / e2e_fp64["value"]
                                          if e2e and e2e_fp64 else None),
                       "algorithm": "the same Morton sort and culled grid as the certified "
                                    "mode, every facet test in FP64"},
        "precision": {"env_facet_tests": cst["env_facet_tests"],
                      "env_facet_fp64": cst["env_facet_fp64"],
                      "env_recheck_fraction": cst["env_facet_fp64"] / max(1, cst["env_facet_tests"]),
                      "amips_tets": cst["amips_tets"], "amips_fp64": cst["amips_fp64"],
                      "amips_recheck_fraction": cst["amips_fp64"] / max(1, cst["amips_tets"]),
                      "exact_orientations": cst["exact_orientations"]},
        "roofline": {"bound": "hbm", "kernel": dom["kernel"], "achieved": achieved,
                     "peak": hbm_peak, "unit": "GB/s", "frac": achieved / hbm_peak,
                     "traffic": traffic_bytes, "peak_source": f"{peak_kind} hbm_gbs",
                     "algorithmic_bytes_per_unit": dom["per_unit"]},
        "roofline_other": roof_other,
        "fp64_pipe": {"kernel": "k_amips_soa (plain FP64, reference energy form)",
                      "achieved_tops": fp64_achieved,
                      "peak_tops_measured": fp64_tflops / 2,
                      "frac": fp64_achieved / (fp64_tflops / 2),
                      "ops_per_tet": flops_per_tet, "fma_peak_tflops_measured": fp64_tflops,
                      "fp32_peak_tflops_measured": fp32_tflops,
                      "note": "binary64 instructions/s against the measured FMA issue rate "
                              "(half the FMA flop rate): no FP contraction, one op each"},
        "e2e": e2e,
        "gpu_launches": 6 * args.steps,
        "gpu_launches_note": "per step: k_amips_soa_cert_bulk, k_amips_recheck, k_point_bins_cid, "
                             "k_point_place_rec, k_env_points_bins, k_env_points_bins_recheck (+ three "
                             "memsets and a CUB scan of the bin counts)",
        "clocks": cert["clocks"],
        "wall_s_timed": cert["wall"],
    }
    # the star-batch and serving configurations are single-GPU workloads: under
    # torchrun (N > 1) the line carries the scaled step only
    if not args.no_batching and ws == 1:
        line["batching"] = run_batching(ctx, V, F, args, dev, ws)
    if not args.no_serving and ws == 1:
        line["serving"] = run_serving(args, dev)
    if rank == 0 and ws == 1 and not args.no_cpu:
        from oracle.oracle import default_threads

        line["cpu_baseline"] = cpu_baseline(T, V, F, P, default_threads())
        line["cpu_baseline"].pop("seconds", None)
        # the reference's own setting (it has no threads): one thread on a bounded
        # sample (1/16 of the step)
        line["cpu_baseline_1thread"] = cpu_baseline(T, V, F, P, 1, frac=16)
        line["cpu_baseline_1thread"].pop("seconds", None)
    if rank == 0:
        print(json.dumps(line), flush=True)
    ctx.close()
    if ws > 1:
        import torch.distributed as dist

        dist.destroy_process_group()
    return 0


N_STARS = 200_000
STAR_SURFACE_FRACTION = 0.5


def run_batching(ctx, V, F, args, dev, ws):
    """Batching workload: one smoothing pass over 200,000 independent stars (half interior,
    half on the 100k-tri displaced sphere), tets per star Poisson(24) clamped to [4, 96] (surface
    stars [6, 96]); one Newton step with at most 8 backtracking trials, inversion checks, and
    for surface stars the projection, quality and one-ring face-envelope checks.  The pass is
    autotuned over the launch shapes, captured in a CUDA graph and replayed; every replay is
    timed with CUDA events on the context stream.  Both precision modes are checked against the
    oracle over the whole batch (status and position bit for bit), and the oracle pass is timed
    on the host cores beside it."""
    import torch

    import tetwild_gb300 as tw
    from oracle.oracle import Oracle, default_threads
    from tetwild_gb300 import synthetic as syn

    xyz, off, tets, ff, cen, kinds = syn.mixed_star_batch(V, F, args.stars, EPS, seed=11,
                                                          surface_fraction=STAR_SURFACE_FRACTION)
    ns, nt = int(cen.size), int(len(tets))
    sd = EPS / 2
    ctx.set_params(EPS * EPS, sd, 1, 8)
    ctx.mesh_upload(xyz)
    d = torch.device(f"cuda:{dev}")
    dev_arr = {k: torch.from_numpy(np.ascontiguousarray(v)).to(d)
               for k, v in dict(off=off.astype(np.int32), tets=tets.astype(np.int32).reshape(-1),
                                ff=ff.astype(np.uint8), cen=cen.astype(np.int32),
                                kinds=kinds.astype(np.uint8)).items()}
    d_out = torch.empty(3 * ns, dtype=torch.float64, device=d)
    d_st = torch.empty(ns, dtype=torch.uint8, device=d)
    a = (dev_arr["off"].data_ptr(), dev_arr["tets"].data_ptr(), dev_arr["ff"].data_ptr(),
         dev_arr["cen"].data_ptr(), dev_arr["kinds"].data_ptr(), ns, nt, d_out.data_ptr(),
         d_st.data_ptr())
    torch.cuda.synchronize()

    nthreads = default_threads()
    o = Oracle()
    S = o.surface(V, F)
    t0 = time.perf_counter()
    want, wst = o.smooth_stars(xyz, off, tets, cen, ff, kinds, surface=S, boundary=S,
                               eps2=EPS * EPS, sd=sd, max_step=1, max_it=8, nthreads=nthreads)
    cpu_s = time.perf_counter() - t0

    stream = torch.cuda.ExternalStream(ctx.stream(), device=f"cuda:{dev}")
    modes = {}
    for name, prec in (("fp32_certified", tw.TW_PRECISION_FP32_CERTIFIED),
                       ("fp64", tw.TW_PRECISION_FP64)):
        ctx.set_precision(prec)
        best, ms_shapes = ctx.smooth_autotune_device(*a)
        ctx.synchronize()
        ctx.capture_begin()
        ctx.smooth_stars_device(*a)
        g = ctx.capture_end()
        for _ in range(max(3, args.warmup)):
            g.launch()
        ctx.synchronize()
        st = d_st.cpu().numpy().astype(np.int8)
        out = d_out.cpu().numpy().reshape(-1, 3)
        mism = {"status": int((st != wst).sum()),
                "position": int(np.any(out != want, axis=1).sum())}
        ctx.reset_stats()
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
               for _ in range(args.steps)]
        barrier(ws)
        for k in range(args.steps):
            evs[k][0].record(stream)
            g.launch()
            evs[k][1].record(stream)
        ctx.synchronize()
        ms = [e0.elapsed_time(e1) for e0, e1 in evs]
        g.close()
        cst = ctx.stats()
        dev_ms = max_over_ranks(sum(ms), ws) / args.steps
        modes[name] = {"stars_per_s": ws * ns / (dev_ms * 1e-3), "ms_per_pass": dev_ms,
                       "p50_ms": float(np.percentile(ms, 50)), "p99_ms": float(np.percentile(ms, 99)),
                       "autotuned_shape": best, "shape_ms": ms_shapes, "mismatches": mism,
                       "env_facet_tests": cst["env_facet_tests"],
                       "env_recheck_fraction": cst["env_facet_fp64"] / max(1, cst["env_facet_tests"])}
    ctx.set_precision(tw.TW_PRECISION_FP32_CERTIFIED)
    counts = np.bincount(wst.astype(np.int64), minlength=6)
    return {
        "workload": f"one smoothing pass over {ns} independent stars ({int((kinds == 0).sum())} "
                    f"interior, {int((kinds == 1).sum())} surface on the 100k-tri displaced sphere), "
                    "tets/star Poisson(24) clamped; Newton max_step 1, max_it 8; projection, "
                    "inversion, quality and face-envelope checks (eps 1e-3, sampling_dist 5e-4); "
                    "autotuned launch shape, CUDA-graph replay",
        "stars": ns, "tets": nt, "value": modes["fp32_certified"]["stars_per_s"],
        "unit": "stars/s", "modes": modes,
        "speedup_certified_vs_fp64": (modes["fp32_certified"]["stars_per_s"] /
                                      modes["fp64"]["stars_per_s"]),
        "oracle_status_counts": {"invalid": int(counts[0]), "not_moved": int(counts[1]),
                                 "moved": int(counts[2]), "reject_flip": int(counts[3]),
                                 "reject_quality": int(counts[4]), "reject_envelope": int(counts[5])},
        "gpu_launches_per_pass": 6,
        "cpu_baseline": {"value": ns / cpu_s, "unit": "stars/s", "cores": nthreads, "kind": "port",
                         "sample": f"the whole pass ({ns} stars) through the oracle"},
    }


N_JOBS = 64
SERVE_SECONDS = 6.0
SERVE_LANES = 4
SERVE_BUDGET = 150 << 30
SERVE_MIX = (("points", 0.40, 1_000, 500_000), ("amips", 0.30, 1_000, 500_000),
             ("faces", 0.15, 1_000, 20_000), ("smooth", 0.15, 1_000, 10_000))
SERVE_SLOTS = 64


def _serving_surface(shape, target, seed):
    from tetwild_gb300 import synthetic as syn

    if shape == 0:
        subdiv = int(np.clip(round(np.log(target / 20.0) / np.log(4.0)), 2, 6))
        return syn.icosphere(subdiv, seed=seed)
    if shape == 1:
        m = max(8, int(round(np.sqrt(target / 6.0))))
        return syn.torus(1.0, 0.3, 3 * m, m)
    r = max(8, int(round(np.sqrt(target / 4.0))))
    return syn.displaced_sphere(seed=seed, n_lon=2 * r, n_rings=r)


def _faces_near(V, F, n, sd, rng):
    """Small triangles (edges ~3 sampling distances) around surface points, offset along the
    normal by U(-1.5, 1.5) eps (eps = sd here)."""
    from tetwild_gb300 import synthetic as syn

    P = syn.envelope_points(V, F, n, 0.0, seed=int(rng.integers(1 << 30)))
    a = rng.normal(size=(n, 3))
    b = rng.normal(size=(n, 3))
    a *= 3 * sd / np.linalg.norm(a, axis=1, keepdims=True)
    b *= 3 * sd / np.linalg.norm(b, axis=1, keepdims=True)
    off = rng.uniform(-1.5, 1.5, (n, 1)) * sd * np.array([[0.0, 0.0, 1.0]])
    return np.hstack([P + off, P + a + off, P + b + off])


def run_serving(args, dev):
    """Serving workload: 64 meshing jobs (icospheres, tori R=1 r=0.3, displaced spheres) of
    1k-200k triangles (log-uniform) resident in HBM under a 150 GB budget; requests of 1k-500k
    queries (log-uniform per kind: envelope points, AMIPS E/J/H, envelope faces, smoothing
    stars) for uniformly chosen jobs.  A burst of 256 requests (the median of three) measures
    capacity in each precision mode; then requests arrive as a Poisson process at 70% of the certified capacity
    for SERVE_SECONDS, and the server-side latency of each (submit to results in host memory)
    gives p50 / p99."""
    import threading

    import tetwild_gb300 as tw
    from tetwild_gb300 import synthetic as syn

    rng = np.random.default_rng(2025)
    sizes = np.exp(rng.uniform(np.log(1e3), np.log(2e5), N_JOBS))
    srv = tw.Server(dev, SERVE_BUDGET, lanes=SERVE_LANES)
    max_n = {k: hi for k, _, _, hi in SERVE_MIX}
    pinned = []

    def pin(a):
        p = tw.PinnedArray(a.shape, a.dtype)
        p.array[...] = a
        pinned.append(p)
        return p.array

    jobs, tris = [], 0
    t_gen = time.perf_counter()
    for i in range(N_JOBS):
        V, F = _serving_surface(i % 3, sizes[i], seed=i)
        tris += len(F)
        diag = float(np.linalg.norm(V.max(0) - V.min(0)))
        eps = 1e-3 * diag
        sd = eps
        j = srv.job_open(V, F, eps * eps, sd)
        if j is None:
            raise RuntimeError("job not admitted under the 150 GB budget")
        P = pin(syn.envelope_points(V, F, max_n["points"], eps, seed=1000 + i))
        Fc = pin(_faces_near(V, F, max_n["faces"], sd, rng))
        xyz, off, tets, ff, cen = syn.surface_star_batch(V, F, max_n["smooth"], eps, seed=2000 + i,
                                                         radius=6 * eps)
        srv.job_mesh(j, xyz)
        jobs.append({"id": j, "P": P, "F": Fc, "off": pin(off), "tets": pin(tets), "ff": pin(ff),
                     "cen": pin(cen), "kinds": pin(np.ones(len(cen), np.uint8))})
    # AMIPS requests take one of 16 log-spaced sizes, each a contiguous pinned SoA batch
    amips_sizes = np.unique(np.geomspace(1_000, max_n["amips"], 16).astype(np.int64))
    Tpool = {int(n): pin(syn.energy_batch(int(n), seed=77 + k)) for k, n in enumerate(amips_sizes)}
    t_gen = time.perf_counter() - t_gen

    # output slots (pinned), reused once the request that held them has completed
    outs = {"points": pin(np.zeros((SERVE_SLOTS, max_n["points"]), np.uint8)),
            "faces": pin(np.zeros((SERVE_SLOTS, max_n["faces"]), np.uint8)),
            "E": pin(np.zeros((SERVE_SLOTS, max_n["amips"]))),
            "J": pin(np.zeros((SERVE_SLOTS, 3 * max_n["amips"]))),
            "H": pin(np.zeros((SERVE_SLOTS, 9 * max_n["amips"]))),
            "flip": pin(np.zeros((SERVE_SLOTS, max_n["amips"]), np.uint8)),
            "sout": pin(np.zeros((SERVE_SLOTS, 3 * max_n["smooth"]))),
            "sst": pin(np.zeros((SERVE_SLOTS, max_n["smooth"]), np.uint8))}

    kinds = [k for k, _, _, _ in SERVE_MIX]
    probs = np.array([p for _, p, _, _ in SERVE_MIX])

    def draw(m):
        out = []
        for _ in range(m):
            k = int(rng.choice(len(kinds), p=probs))
            _, _, lo, hi = SERVE_MIX[k]
            n = int(np.exp(rng.uniform(np.log(lo), np.log(hi))))
            if kinds[k] == "amips":
                n = int(amips_sizes[np.argmin(np.abs(np.log(amips_sizes / n)))])
            out.append((kinds[k], int(rng.integers(N_JOBS)), n))
        return out

    def submit(i, req):
        kind, ji, n = req
        J = jobs[ji]
        slot = i % SERVE_SLOTS
        if kind == "points":
            t, _ = srv.submit_points(J["id"], J["P"][:n], out=outs["points"][slot, :n])
        elif kind == "faces":
            t, _ = srv.submit_faces(J["id"], J["F"][:n], out=outs["faces"][slot, :n])
        elif kind == "amips":
            o = (outs["E"][slot, :n], outs["J"][slot, :3 * n].reshape(3, n),
                 outs["H"][slot, :9 * n].reshape(9, n), outs["flip"][slot, :n])
            t, _ = srv.submit_amips(J["id"], Tpool[n], out=o)
        else:
            o = (outs["sout"][slot, :3 * n].reshape(n, 3), outs["sst"][slot, :n])
            t, _ = srv.submit_smooth(J["id"], J["off"][:n + 1], J["tets"][:J["off"][n]],
                                     J["cen"][:n], J["ff"][:J["off"][n]], J["kinds"][:n], out=o)
        return t

    def run(reqs, arrivals=None):
        """Submits reqs (at the given arrival times, else at once) and returns per-request
        latencies (ms) and the wall time from the first submission to the last completion."""
        lat = [0.0] * len(reqs)
        done = [threading.Event() for _ in reqs]
        tickets = [None] * len(reqs)
        ready = [threading.Event() for _ in reqs]
        err = []

        def waiter():
            try:
                for i in range(len(reqs)):
                    ready[i].wait()
                    lat[i] = srv.wait(tickets[i], 120.0)
                    done[i].set()
            except Exception as e:
                err.append(e)
                for d in done:
                    d.set()

        th = threading.Thread(target=waiter)
        th.start()
        t0 = time.perf_counter()
        for i, r in enumerate(reqs):
            if i >= SERVE_SLOTS:
                done[i - SERVE_SLOTS].wait()
            if arrivals is not None:
                dt = t0 + arrivals[i] - time.perf_counter()
                if dt > 0:
                    time.sleep(dt)
            tickets[i] = submit(i, r)
            ready[i].set()
        th.join()
        wall = time.perf_counter() - t0
        if err:
            raise err[0]
        return lat, wall

    burst = draw(256)
    q_burst = sum(n for _, _, n in burst)
    cap = {}
    for name, prec in (("fp64", tw.TW_PRECISION_FP64),
                       ("fp32_certified", tw.TW_PRECISION_FP32_CERTIFIED)):
        srv.set_params(prec, 1, 8)
        run(burst[:32])                     # warm-up: lane scratch grows to size
        # the median of three bursts (one burst lasts tens of ms: host jitter shows)
        runs = sorted((run(burst) for _ in range(3)), key=lambda r: r[1])
        lat, wall = runs[1]
        cap[name] = {"queries_per_s": q_burst / wall, "requests_per_s": len(burst) / wall,
                     "wall_s": wall, "walls_s": [r[1] for r in runs],
                     "p50_ms": float(np.percentile(lat, 50)),
                     "p99_ms": float(np.percentile(lat, 99))}
    rate = 0.7 * cap["fp32_certified"]["requests_per_s"]
    m = max(64, int(rate * SERVE_SECONDS))
    reqs = draw(m)
    arrivals = np.cumsum(rng.exponential(1.0 / rate, m))
    st0 = srv.stats()
    lat, wall = run(reqs, arrivals)
    st1 = srv.stats()
    q = sum(n for _, _, n in reqs)
    by_kind = {}
    for k in kinds:
        l = [x for x, r in zip(lat, reqs) if r[0] == k]
        if l:
            by_kind[k] = {"requests": len(l), "p50_ms": float(np.percentile(l, 50)),
                          "p99_ms": float(np.percentile(l, 99))}
    stats = srv.stats()
    srv.close()
    for p_ in pinned:
        p_.free()
    return {
        "workload": f"{N_JOBS} jobs (icosphere / torus R=1 r=0.3 / displaced sphere, "
                    f"1k-200k tris log-uniform, {tris} tris in all) under a 150 GB budget; "
                    "requests: points 40% (1k-500k), AMIPS E/J/H 30% (16 log-spaced sizes 1k-500k), faces 15% "
                    "(1k-20k), smoothing stars 15% (1k-10k), log-uniform sizes, uniform jobs; "
                    f"{SERVE_LANES} lanes; certified FP32 mode",
        "arrival_rate_per_s": rate, "offered_load": "70% of the certified burst capacity",
        "requests": m, "queries": q, "seconds": wall,
        "queries_per_s": q / wall, "unit": "queries/s",
        "p50_ms": float(np.percentile(lat, 50)), "p99_ms": float(np.percentile(lat, 99)),
        "latency_by_kind": by_kind,
        "burst_capacity": cap,
        "capacity_speedup_certified_vs_fp64": (cap["fp32_certified"]["queries_per_s"] /
                                               cap["fp64"]["queries_per_s"]),
        "batches": st1["batches"] - st0["batches"],
        "mean_requests_per_batch": m / max(1, st1["batches"] - st0["batches"]),
        "max_requests_per_batch": stats["max_requests_per_batch"],
        "hbm_bytes_used": stats["bytes_used"], "setup_s": t_gen,
    }


def barrier(ws):
    if ws > 1:
        import torch.distributed as dist

        dist.barrier()


def max_over_ranks(x, ws):
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist

    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def check_sample(T, P, V, F, dE, dFl, dO, n=20000):
    """Decision mismatches vs the oracle on a strided sample of this step's outputs."""
    from oracle.oracle import Oracle, default_threads

    o = Oracle()
    idx = np.linspace(0, N_TETS - 1, n).astype(np.int64)
    Ts = np.ascontiguousarray(T[:, idx])
    E, _, _, Fo = o.amips_batch_soa(Ts, quality=True, nthreads=default_threads(), jacobian=False,
                                    hessian=False)
    gE = dE.cpu().numpy()[idx]
    gF = dFl.cpu().numpy()[idx]
    pidx = np.linspace(0, N_POINTS - 1, n).astype(np.int64)
    Po = o.surface(V, F).points_out(np.ascontiguousarray(P[pidx]), EPS * EPS,
                                    nthreads=default_threads())
    gO = dO.cpu().numpy()[pidx]
    fin = E < 1e50
    sentinel_mismatch = int(((gE >= 1e50) != ~fin).sum())
    rel = np.abs(gE[fin] - E[fin]) / np.abs(E[fin]) if fin.any() else np.zeros(1)
    return {"sampled": 2 * n, "flip": int((gF != Fo).sum()),
            "energy_sentinel": sentinel_mismatch, "envelope": int((gO != Po).sum()),
            "energy_max_rel_err_vs_fp64": float(rel.max()),
            "energy_bit_identical_fraction": float((gE == E).mean())}


def run_e2e(ctx, T, P, args, ws, steps=None):
    """The step through the C-ABI host calls (tw_amips_soa, tw_envelope_points) with
    pinned host buffers, in the context's current precision mode."""
    import tetwild_gb300 as tw

    steps = steps or args.steps
    hT = tw.PinnedArray(T.shape, np.float64)
    hT.array[...] = T
    hP = tw.PinnedArray(P.shape, np.float64)
    hP.array[...] = P
    oE = tw.PinnedArray((N_TETS,), np.float64)
    oJ = tw.PinnedArray((3, N_TETS), np.float64)
    oH = tw.PinnedArray((9, N_TETS), np.float64)
    oF = tw.PinnedArray((N_TETS,), np.uint8)
    oO = tw.PinnedArray((N_POINTS,), np.uint8)
    lib, h = ctx.lib, ctx.h

    def step():
        st = lib.tw_amips_soa(h, hT.array.ctypes.data, N_TETS, tw.TW_ENERGY_QUALITY,
                              oE.array.ctypes.data, oJ.array.ctypes.data, oH.array.ctypes.data,
                              oF.array.ctypes.data)
        assert st == 0, st
        st = lib.tw_envelope_points(h, hP.array.ctypes.data, N_POINTS, tw.TW_SURFACE_INPUT,
                                    oO.array.ctypes.data)
        assert st == 0, st

    for _ in range(max(1, min(args.warmup, 3))):
        step()
    barrier(ws)
    t0 = time.perf_counter()
    for _ in range(steps):
        step()
    dt = time.perf_counter() - t0
    dt = max_over_ranks(dt, ws)
    for a in (hT, hP, oE, oJ, oH, oF, oO):
        a.free()
    q = (N_TETS + N_POINTS) * steps * ws
    return {"value": q / dt, "unit": UNIT, "h2d_bytes_per_step": 96 * N_TETS + 24 * N_POINTS,
            "d2h_bytes_per_step": (8 + 24 + 72 + 1) * N_TETS + N_POINTS,
            "ms_per_step": 1e3 * dt / steps, "steps": steps}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--no-e2e", action="store_true", help="skip the host-buffer leg")
    ap.add_argument("--no-batching", action="store_true", help="skip the star-batch pass")
    ap.add_argument("--no-serving", action="store_true", help="skip the serving loop")
    ap.add_argument("--only-batching", action="store_true",
                    help="profiling: the star-batch pass alone, no benchmark line")
    ap.add_argument("--stars", type=int, default=N_STARS, help="smaller star batch for profiling only")
    ap.add_argument("--modes", default="plain,cert",
                    help="profiling runs may time one mode only (then no benchmark line)")
    ap.add_argument("--tets", type=int, default=N_TETS, help="smaller case for profiling only")
    ap.add_argument("--points", type=int, default=N_POINTS, help="smaller case for profiling only")
    ap.add_argument("--bin-cell", type=float, default=None,
                    help="TW_TUNE_BIN_CELL for the step (0: the point test reads the grid's "
                         "hashed cells instead of the bin index); profiling only")
    args = ap.parse_args()
    set_sizes(args.tets, args.points)
    if args.impl == "reference":
        return run_reference(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
