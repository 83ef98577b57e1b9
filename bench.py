"""Benchmark: ImplicitSteady time-to-steady and DVM cell-velocity updates/s of the UGKS2D hot path on B200.

Workload (one "step" of this script): the reference's delivered ImplicitSteady Couette case
(8x64 cells, 32x32 velocities velocity_half32_scale2, CFL 0.1, nCFL 1000, omega 0.5, Kn 0.1, mass
rescale on, FP64) solved from the cold start (uniform Maxwellian rho=1, T=1, u=0) until the
five-state gate passes (residual tolerance 1e-8, moment 1e-12, 5 consecutive accepted states).
One update = one (cell, velocity) with both h and b advanced by one pseudo-step; a solve is
8*64*1024 * (pseudo-steps to the gate) updates.  Inputs are synthetic (the cold start the case
itself prescribes), no dataset is involved.

  value          device-resident throughput over the K timed solves (CUDA events on the solver's
                 stream, max over ranks); time_to_steady_s = mean seconds per solve.
  e2e            the same through the public C ABI with host buffers: every solve uploads h, b, W
                 from pinned host memory, runs to the gate and downloads the final state.
  roofline       the dominant stage of the pseudo-step (per-stage CUDA events in a separate
                 profiling pass, same stream) against its algorithmic bytes.
  fp64           algorithmic FP64 operations per update (counted by oracle/count_flops.py: the reference's
                 formulation's) x updates/s, beside a cuBLAS float64 GEMM measured in the same run.  In the
                 roofline, whose kernels do those operations, also as a fraction of it; in the other
                 methods' objects the kernels need fewer for the same update (tensor-product velocity
                 tables), so there it is a rate of finished work and no fraction is formed.
  cpu_baseline   the C oracle (a restatement of the reference's Fortran; the Fortran itself does not
                 build on this image) timed on a bounded number of pseudo-steps of the same case.
  explicit_plain the plain second-order Explicit step (1000 steps, CFL 0.5, omega 0.81) for context.
  high_order_implicit  HighOrderImplicit (WENO5-AO S2 evolution + LU-SGS) from the cold start to its
                 3000-pseudo-step cap, c_minus_1 recorded, with a bounded oracle sample beside it.
  s2cn2          the explicit high-order S2CN2 step (S2 evolution + Crank-Nicolson collision) on the same
                 case, with a bounded oracle sample beside it.
  adjoint        the adjoint config's cases (8x64x1024): the gradient of the wall outputs by the discrete
                 adjoint (checkpointed forward + reverse sweep), timed against the plain forward of the same cases.
  batched        (N > 1: the instances are split over the ranks by an LPT greedy on cells x velocities,
                 no collective; time = max over ranks; value = all instances' work / that time)
                 256 S2CN2 instances of the batched distribution (Kn log-uniform in [0.01, 1], wall Mach
                 in [0.5, 3], wall temperature ratio in [0.8, 1.2], 8x{32,64,128} cells, {24,32,48}^2
                 velocities, PCG64(20261203)) advanced together (one graph launch per two steps, stream
                 count picked by the autotuner); aggregate updates/s and the ratio to s2cn2's plain rate.

Multi-GPU: a single instance does not shard (one domain per GPU); N ranks run N independent
replicas ("scaling": "weak").  --impl reference times the CPU restatement of the reference on host
cores on the same workload.
"""
import argparse
import gc
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "DVM cell·vel updates/s + time-to-steady on 1 B200, batched vs plain, vs CPU ref"
UNIT = "cell·vel updates/s"
MAX_PSEUDO_STEPS = 3000
TOL10_MAX_PSEUDO_STEPS = 20000
EXPLICIT_STEPS = 1000
HO_MAX_PSEUDO_STEPS = 3000     # HighOrderImplicit cap (cases/high_implicit/Config.ini MAX_ITER)
S2CN2_STEPS = 400
REFINED_PSEUDO_STEPS = 100   # timed pseudo-steps of the refined HighOrderImplicit variant
BATCH_STEPS = 4               # batched steps timed (each advances all 256 instances by one step)
ADJ_STEPS = 50                # adjoint timing: one checkpoint segment of 50 steps per case
ADJ_EVERY = 50
ADJ_CASES = 4                 # cases of the 64 timed (each gradient is an independent instance)
ADJ_LONG_STEPS = 200          # and four segments of the first case: the per-step cost of a long run
C5_STEPS = 2                  # steps timed at the adjoint config's shape (64 cases, 8x64x1024); even:
                              # one replay of the two-step graph
# algorithmic bytes per cell*velocity of the stages (FP64 h and b):
#   lusgs_forward  reads the right-hand side (h, b) and writes the correction (h, b)      32 B
#   lusgs_backward also reads the forward correction                                   48 B
#   post_residual  reads h, b, the x- and y-face fluxes (h, b) and writes stream (h, b)   80 B
#   post_fluxes    reads h, b and their slopes, writes the face fluxes                   64 B
#   explicit step  reads h, b, writes h, b                                              32 B
# accepted pseudo-steps of the delivered ImplicitSteady case to its five-state gate on the B200 (the C
# oracle stops at the same step; the reference's own run stopped at 1096): the reference arm, which
# samples pseudo-steps, extrapolates its time to steady with it
PSEUDO_STEPS_TO_GATE = 1097
BYTES_PER_UPDATE_PSEUDO_STEP = 240   # compulsory traffic of one implicit pseudo-step per cell*velocity
# DRAM bytes (read + write) of one ImplicitSteady pseudo-step at 8x64x1024: the sum over its launches in
# the ncu launch list of 16 pseudo-steps (dram__bytes_read.sum + dram__bytes_write.sum, 289 launches,
# init kernels excluded).  ncu flushes the caches before every launch, so this is the cold-cache upper
# bound of the graph-replayed step, in which the 8.4 MB state and the work arrays stay in L2.
TRAFFIC_PER_PSEUDO_STEP_8X64X1024 = 149_164_656
STAGE_BYTES_PER_UPDATE = {"lusgs_forward": 32, "lusgs_backward": 48, "post_residual": 80, "post_fluxes": 64}
BYTES_PER_UPDATE_EXPLICIT = 32
# pr2_sweep works on the macroscopic fields: per cell W, X, rate, gamma (4 each), two 16-value face
# flux tables, and writes Y (4): 52 doubles per cell per launch
PR2_BYTES_PER_CELL = 52 * 8
# Algorithmic FP64 operations per cell*velocity update (add/sub + mul + div + sqrt), counted by the
# op-counting build of the oracle on the 8x64x1024 cases (python oracle/count_flops.py).  The
# implicit pseudo-steps count one evaluation less than the reference runs: the device reuses the
# accepted-state evaluation as the next pre-update one (reference: 3568 and 58725).
GRAPH_PROFILE_STEPS = 96   # pseudo-steps of the graph-mode stage timing (12 batch graphs of 8)
VARIANT_STEPS = 40   # timed steps of each research wall variant (8x64x1024, after 4 warm-up steps)
FLOPS_PER_UPDATE = {"explicit": 1565.9, "implicit_steady": 2211.5, "high_order_implicit": 29736.7, "s2cn2": 29241.7}
# S2CN2 per velocity set (oracle/count_flops.py: S2CN2_24, S2CN2 (32^2), S2CN2_48 on the 8x64 case)
S2CN2_FLOPS_BY_TABLE = {24: 29306.5, 32: 29241.7, 48: 27542.5}
WORKLOAD = ("ImplicitSteady 2nd-order UGKS Couette 8x64 cells, 32x32 velocities (velocity_half32_scale2), "
            "CFL 0.1, nCFL 1000, Kn 0.1, mass rescale on, cold start to the five-state gate (tol 1e-8)")


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def fp64_peak(device):
    """FP64 throughput of this GPU in TFLOP/s: a cuBLAS float64 GEMM (8192^3) through torch, the
    denominator of the FP64 fraction (B200's nominal FP64 and FP64 tensor peaks are both 37 TFLOP/s)."""
    import torch
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device=device)
    b = torch.randn(n, n, dtype=torch.float64, device=device)
    for _ in range(2):
        torch.matmul(a, b)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(5):
        torch.matmul(a, b)
    e1.record()
    e1.synchronize()
    t = e0.elapsed_time(e1) * 1e-3 / 5
    del a, b
    torch.cuda.empty_cache()
    return 2.0 * n ** 3 / t / 1e12


def fp64_fraction(flops_per_update, updates_per_s, peak_tflops):
    """For kernels that do the counted operations."""
    achieved = flops_per_update * updates_per_s / 1e12
    return {"flops_per_update": flops_per_update, "achieved_tflops": achieved, "peak_tflops": peak_tflops,
            "frac": achieved / peak_tflops, "peak_source": "cuBLAS float64 GEMM 8192^3 measured in this run"}


def fp64_reference_work(flops_per_update, updates_per_s, gemm_tflops):
    """For kernels that finish the same update with fewer operations: the reference formulation's operations in the
    time taken, which is no rate of the hardware and no fraction of its peak."""
    return {"reference_flops_per_update": flops_per_update, "reference_work_tflops": flops_per_update * updates_per_s / 1e12,
            "gemm_tflops": gemm_tflops, "gemm_source": "cuBLAS float64 GEMM 8192^3 measured in this run",
            "counted": "the reference formulation's operations; the kernels do fewer on tensor-product tables"}


class ClockSampler:
    """SM clocks and clock-event (throttle) reasons sampled during the timed region.

    NVML (the library nvidia-smi is built on) is polled from a host thread every `period` s;
    `nvidia-smi -lms` is the alternative (--sampler smi).  Reasons recorded: hw_slowdown,
    hw_thermal_slowdown, sw_thermal_slowdown, sw_power_cap.
    """

    REASONS = {"hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40, "sw_power_cap": 0x4}

    def __init__(self, index, kind="nvml", period=0.2):
        self.index, self.kind, self.period = index, kind, period
        self.samples, self.reasons, self.smax = [], set(), None
        self._stop = threading.Event()
        self._lock = threading.Lock()
        self.proc = None
        self.lines = []

    def begin(self):
        """Start of the timed window: the samples and reasons taken so far (the sampler runs from before
        the warm-up, so its start-up is not inside the window) are dropped."""
        with self._lock:
            self.samples, self.reasons = [], set()
        if self.kind == "nvml" and getattr(self, "nv", None):
            self._poll_once()   # a sample at the window's start, whatever the polling phase

    def start(self):
        if self.kind == "none":
            return
        if self.kind == "smi":
            q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
                 "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                 "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
            try:
                self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                                              "--format=csv,noheader,nounits", "-lms", str(int(self.period * 1000))],
                                             stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
                self.t = threading.Thread(target=self._read_smi, daemon=True)
                self.t.start()
            except Exception:
                self.proc = None
            return
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(self.index)
            self.smax = float(pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM))
        except Exception:
            self.nv = None
            return
        self.t = threading.Thread(target=self._poll_nvml, daemon=True)
        self.t.start()

    def _poll_once(self):
        nv = self.nv
        try:
            mhz = float(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM))
            mask = nv.nvmlDeviceGetCurrentClocksEventReasons(self.h)
            with self._lock:
                self.samples.append(mhz)
                for name, bit in self.REASONS.items():
                    if mask & bit:
                        self.reasons.add(name)
        except Exception:
            pass

    def _poll_nvml(self):
        while not self._stop.is_set():
            self._poll_once()
            self._stop.wait(self.period)

    def _read_smi(self):
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.proc.stdout:
            parts = [p.strip() for p in line.strip().split(",")]
            if len(parts) < 9:
                continue
            try:
                mhz, self.smax = float(parts[1]), float(parts[2])
            except ValueError:
                continue
            with self._lock:
                self.samples.append(mhz)
                for n, v in zip(names, parts[5:9]):
                    if v.lower().startswith("active"):
                        self.reasons.add(n)

    def stop(self):
        if self.kind == "none":
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "sampler": "none"}
        self._stop.set()
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
        elif getattr(self, "t", None):
            self.t.join(timeout=2)
        return {"sm_mhz": statistics.median(self.samples) if self.samples else None, "sm_max_mhz": self.smax,
                "reasons": sorted(self.reasons), "samples": len(self.samples),
                "sampler": "nvml" if self.kind == "nvml" else "nvidia-smi"}


def dist_env():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


def host_cpu():
    """The host CPU the baselines ran on: the model name of /proc/cpuinfo (what lscpu prints) and the
    logical CPUs of the host."""
    model = "unknown"
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.lower().startswith("model name"):
                    model = line.split(":", 1)[1].strip()
                    break
    except OSError:
        pass
    return {"cpu_model": model, "host_cpus": os.cpu_count()}


def cpu_baseline(case, velocity, nsteps=30, threads=None):
    """The oracle (single-domain restatement of the reference Fortran) on `nsteps` pseudo-steps."""
    from oracle.oracle import Oracle, set_threads
    nthreads = set_threads(threads)
    o = Oracle(case, *velocity)
    o.init_freestream()
    o.implicit_init()
    o.implicit_step()   # warm-up
    t0 = time.perf_counter()
    for _ in range(nsteps):
        o.implicit_step()
    el = time.perf_counter() - t0
    units = case.nx * case.ny * len(velocity[0]) * nsteps
    return {"value": units / el, "unit": UNIT, "cores": nthreads, "kind": "port", **host_cpu(),
            "seconds_per_pseudo_step": el / nsteps,
            "sample": f"{nsteps} ImplicitSteady pseudo-steps of the 8x64x1024 cold start after 1 warm-up step "
                      f"({el:.2f} s, C oracle -O2, {nthreads} pthread(s) over cells, faces and slabs)"}


def cpu_sample_high_order(velocity, nsteps=2, threads=None):
    """The oracle on `nsteps` HighOrderImplicit pseudo-steps of the cold start (after one warm-up step)."""
    from oracle.oracle import Oracle, set_threads
    from ugks2d_high_order_b200.case import reference_case
    nthreads = set_threads(threads)
    case = reference_case("HighOrderImplicit")
    o = Oracle(case, *velocity)
    o.init_freestream()
    o.implicit_init()
    o.implicit_step()
    t0 = time.perf_counter()
    for _ in range(nsteps):
        o.implicit_step()
    el = time.perf_counter() - t0
    units = case.nx * case.ny * len(velocity[0]) * nsteps
    return {"value": units / el, "unit": UNIT, "cores": nthreads, "kind": "port", **host_cpu(),
            "seconds_per_pseudo_step": el / nsteps,
            "sample": f"{nsteps} HighOrderImplicit pseudo-steps of the cold start ({el:.2f} s, C oracle -O2, "
                      f"{nthreads} pthread(s)); the reference's published figure is 1.8153 s per pseudo-step on 8 "
                      f"MPI ranks (analysis.json high_implicit: 5445.8 s for 3000)"}


def cpu_sample_s2cn2(velocity, nsteps=3, threads=None):
    """The oracle on `nsteps` S2CN2 steps of the cold start (after one warm-up step)."""
    from oracle.oracle import Oracle, set_threads
    from ugks2d_high_order_b200.case import reference_case
    nthreads = set_threads(threads)
    case = reference_case("S2CN2")
    o = Oracle(case, *velocity)
    o.init_freestream()
    o.s2cn2_step()
    t0 = time.perf_counter()
    for _ in range(nsteps):
        o.s2cn2_step()
    el = time.perf_counter() - t0
    units = case.nx * case.ny * len(velocity[0]) * nsteps
    return {"value": units / el, "unit": UNIT, "cores": nthreads, "kind": "port", **host_cpu(),
            "seconds_per_step": el / nsteps,
            "sample": f"{nsteps} S2CN2 steps of the cold start ({el:.2f} s, C oracle -O2, {nthreads} pthread(s))"}


def run_reference_arm(args):
    world, rank, _ = dist_env()
    if rank != 0:
        return
    from ugks2d_high_order_b200.case import reference_case, load_velocity_half32
    case = reference_case("ImplicitSteady")
    vel = load_velocity_half32()
    from oracle.oracle import Oracle, set_threads
    nthreads = set_threads(None)
    o = Oracle(case, *vel)
    o.init_freestream()
    o.implicit_init()
    per_step = max(1, int(os.environ.get("UGKS_REF_SAMPLE_STEPS", "10")))
    for _ in range(args.warmup):
        o.implicit_step()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        for _ in range(per_step):
            o.implicit_step()
    el = time.perf_counter() - t0
    units = case.nx * case.ny * len(vel[0]) * per_step * args.steps
    v = units / el
    line = {"metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "impl": "reference",
            "config": {"workload": WORKLOAD, "pseudo_steps_per_bench_step": per_step,
                       "sampled": f"each bench step times {per_step} pseudo-steps of the solve (from the cold "
                                  f"start, {args.warmup * per_step} warm-up pseudo-steps first), not a solve to the "
                                  f"gate; the rate is per cell-velocity update, the unit of the GPU arm's value",
                       "seconds_per_pseudo_step": el / (per_step * args.steps),
                       "time_to_steady_estimate_s": el / (per_step * args.steps) * PSEUDO_STEPS_TO_GATE,
                       "parallelism": "host threads"},
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": nthreads, "kind": "port", **host_cpu(),
                             "sample": f"{per_step} pseudo-steps of the cold start per bench step (the Fortran "
                                       f"reference cannot be built on this image; its C restatement is timed)"},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def run_long(args):
    """The configurations at their full stated length, run once (not part of the default bench, whose
    timed work stays near a minute): the 256-instance batch for its 2000 steps, and the refined
    HighOrderImplicit variant (16x128 cells, 48x48 velocities) to its 3000 pseudo-step cap.  Prints one
    JSON line with "mode": "long"."""
    import torch
    _, _, local = dist_env()
    torch.cuda.set_device(local)
    from ugks2d_high_order_b200.batch import Batch
    from ugks2d_high_order_b200.case import batched_cases, refined_high_order_case, velocity_table
    from ugks2d_high_order_b200.solver import Solver
    out = {"mode": "long"}
    tables = {n: velocity_table(n) for n in (24, 32, 48)}

    # the refined HighOrderImplicit variant from the cold start to the cap
    rcase = refined_high_order_case()
    sr = Solver(rcase, *tables[48], device=local)
    sr.init_freestream()
    sr.implicit_init()
    st = torch.cuda.ExternalStream(sr.stream)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(st):
        e0.record(st)
        done, conv, rep = sr.step_implicit(HO_MAX_PSEUDO_STEPS)
        e1.record(st)
    e1.synchronize()
    ms = e0.elapsed_time(e1)
    sr.close()
    out["refined_high_order_implicit"] = {
        "pseudo_steps": int(done), "converged": bool(conv), "wall_s": ms * 1e-3,
        "ms_per_pseudo_step": ms / max(done, 1),
        "updates_per_s": rcase.nx * rcase.ny * len(tables[48][0]) * done / (ms * 1e-3),
        "c_minus_1": float(rep[52]), "moment": float(rep[1]), "R1_R8": [float(x) for x in rep[4:12]],
        "science_1_4": [float(x) for x in rep[12:16]], "Rh_Rb": [float(rep[24]), float(rep[25])],
        "config": "HighOrderImplicit 16x128 cells, 48x48 velocities (generated half-range table), 8 slabs, "
                  "CFL 0.1, nCFL 1000, mass rescale on, cold start to the 3000 pseudo-step cap"}

    # the batched distribution for its full 2000 steps
    cases = batched_cases()
    bt = Batch([(c, tables[n]) for c, n in cases], device=local, max_streams=32)
    bt.init_freestream()
    k_tuned, _ = bt.tune(steps=2)
    bt.init_freestream()
    bs = torch.cuda.ExternalStream(bt.stream)
    b0, b1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    nsteps = 2000
    with torch.cuda.stream(bs):
        b0.record(bs)
        bdone, bst = bt.run(nsteps)
        b1.record(bs)
    b1.synchronize()
    bms = b0.elapsed_time(b1)
    reps = np.stack([bt.report(i) for i in range(len(cases))])
    kn = np.array([c.mu_ref * np.sqrt(np.pi) for c, _ in cases])
    cv = sum(c.nx * c.ny * n * n for c, n in cases)
    out["batched_full"] = {
        "instances": len(cases), "steps": nsteps, "streams": int(k_tuned),
        "all_accepted": bool((bdone == nsteps).all() and not bst.any()),
        "steps_done_min": int(bdone.min()), "wall_s": bms * 1e-3, "updates_per_s": cv * nsteps / (bms * 1e-3),
        "final_drift_max": float(reps[:, 9].max()), "final_drift_median": float(np.median(reps[:, 9])),
        "final_cnres_max": float(reps[:, 1].max()), "final_mmerr_max": float(reps[:, 2].max()),
        "min_h_min": float(reps[:, 5].min()), "min_b_min": float(reps[:, 7].min()),
        "kn_range": [float(kn.min()), float(kn.max())],
        "config": "256 S2CN2 instances, seed PCG64(20261203), Kn log-uniform [0.01, 1], wall Mach [0.5, 3], "
                  "Tw ratio [0.8, 1.2], 8x{32,64,128} cells, {24,32,48}^2 velocities, CFL 0.1, cold start, "
                  "2000 steps; drift is each instance's conservation drift against its wall ledger at the last "
                  "step (every step is gated at 2e-12)"}
    bt.close()
    print(json.dumps(out), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--sampler", default="nvml", choices=["nvml", "smi", "none"],
                    help="clock sampler during the timed region")
    ap.add_argument("--sampler-period", type=float, default=0.5, help="seconds between clock samples")
    ap.add_argument("--long", action="store_true",
                    help="run the batched and refined configurations once at their full length instead")
    args = ap.parse_args()
    if args.long:
        run_long(args)
        return
    if args.impl == "reference":
        run_reference_arm(args)
        return

    world, rank, local = dist_env()
    import torch
    pg = None
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=timedelta(seconds=120), device_id=torch.device("cuda", local))
        pg = dist
    else:
        torch.cuda.set_device(local)

    from ugks2d_high_order_b200.case import baseline_explicit_case, load_velocity_half32, reference_case
    from ugks2d_high_order_b200.solver import Solver
    case = reference_case("ImplicitSteady")
    vel = load_velocity_half32()
    s = Solver(case, *vel, device=local)
    nc, nv = case.nx * case.ny, len(vel[0])
    stream = torch.cuda.ExternalStream(s.stream)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=f"cuda:{local}")

    def barrier():
        if pg:
            t = torch.zeros(1, device=f"cuda:{local}")
            pg.all_reduce(t)
        torch.cuda.synchronize()

    def max_over_ranks(x):
        if pg:
            t = torch.tensor([x], device=f"cuda:{local}")
            pg.all_reduce(t, op=pg.ReduceOp.MAX)
            x = float(t.item())
        return x

    def solve():
        s.init_freestream()
        s.implicit_init()
        done, conv, rep = s.step_implicit(MAX_PSEUDO_STEPS)
        if not conv:
            raise RuntimeError(f"five-state gate not reached in {MAX_PSEUDO_STEPS} pseudo-steps")
        return done

    # ---------------- device-resident timing: K cold-start solves to the gate
    # The clock sampler starts before the warm-up (its library start-up stays out of the timed window)
    # and keeps only the samples taken inside the window.
    # The collector runs before the warm-up and stays off through the timed window: no collector pause
    # between the solves' host calls, and no idle gap between the warm-up and the timed solves.
    sampler = ClockSampler(local, args.sampler, args.sampler_period)
    sampler.start()
    gc.collect()
    gc.disable()
    with torch.cuda.stream(stream):
        for _ in range(args.warmup):   # as the timed loop, flush included (its first call loads its kernel)
            flush.zero_()
            solve()
    launches0 = s.launch_count
    barrier()
    sampler.begin()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    pseudo = []
    with torch.cuda.stream(stream):
        evs[0].record(stream)
        for k in range(args.steps):
            flush.zero_()          # L2 flush between bench steps (256 MB > 126 MB L2)
            pseudo.append(solve())
            evs[k + 1].record(stream)
    evs[-1].synchronize()
    gc.enable()
    barrier()
    clocks = sampler.stop()
    ms = max_over_ranks(evs[0].elapsed_time(evs[-1]))
    solve_ms = [evs[k].elapsed_time(evs[k + 1]) for k in range(args.steps)]
    launches = s.launch_count - launches0
    units = nc * nv * sum(pseudo)
    value = world * units / (ms * 1e-3)

    # ---------------- end-to-end through the C ABI with pinned host buffers
    s.init_freestream()
    h, b, W = s.download()
    hp = torch.from_numpy(h).pin_memory()
    bp = torch.from_numpy(b).pin_memory()
    Wp = torch.from_numpy(W).pin_memory()
    ho = torch.empty_like(hp).pin_memory()
    bo = torch.empty_like(bp).pin_memory()
    Wo = torch.empty_like(Wp).pin_memory()
    import ctypes
    dp = ctypes.POINTER(ctypes.c_double)
    P = lambda t: ctypes.cast(t.data_ptr(), dp)
    L = s.L
    done_c, conv_c = ctypes.c_int(), ctypes.c_int()
    rep = np.zeros(80)

    def e2e_solve():
        flush.zero_()
        rc = L.ugks_upload_state(s.ctx, P(hp), P(bp), P(Wp))
        rc = rc or L.ugks_implicit_init(s.ctx)
        rc = rc or L.ugks_implicit_steps(s.ctx, MAX_PSEUDO_STEPS, ctypes.byref(done_c), ctypes.byref(conv_c),
                                         rep.ctypes.data_as(dp))
        rc = rc or L.ugks_download_state(s.ctx, P(ho), P(bo), P(Wo))
        if rc or not conv_c.value:
            raise RuntimeError(f"end-to-end solve failed (status {rc}, converged {conv_c.value})")
        return done_c.value

    # as above: the collector off from before one untimed call through the timed window
    gc.collect()
    gc.disable()
    with torch.cuda.stream(stream):
        e2e_solve()
    e_pseudo = 0
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(stream):
        e0.record(stream)
        for _ in range(args.steps):
            e_pseudo += e2e_solve()
        e1.record(stream)
    e1.synchronize()
    gc.enable()
    barrier()
    ems = max_over_ranks(e0.elapsed_time(e1))
    e2e_value = world * nc * nv * e_pseudo / (ems * 1e-3)
    state_bytes = (h.nbytes + b.nbytes + W.nbytes)

    # ---------------- per-stage timing pass (events between stages, no graph)
    s.init_freestream()
    s.implicit_init()
    s.step_implicit(20)
    s.profile(True)
    prof_steps = 100
    s.step_implicit(prof_steps)
    from ugks2d_high_order_b200.capi import IMPLICIT_STAGES
    ustimes = {name: s.profile_read(name) for name in IMPLICIT_STAGES}
    s.profile(False)
    # ... and the same stages as the batch graphs run them: the stage events are captured into the graphs
    # as event nodes, and each 8-step batch's last pseudo-step is timed (no launch gaps of its own)
    s.init_freestream()
    s.implicit_init()
    s.step_implicit(20)
    s.profile(True, graph=True)
    s.step_implicit(GRAPH_PROFILE_STEPS)
    stimes = {name: s.profile_read(name) for name in IMPLICIT_STAGES}
    s.profile(False)
    stot = sum(t for t, _ in stimes.values())
    top = max(stimes, key=lambda k: stimes[k][0])
    t_top, n_top = stimes[top]
    peak, peak_kind = peaks()
    if top == "pr2_sweep":
        n_launch = n_top * case.macro_sweeps
        algo = PR2_BYTES_PER_CELL * nc
        kname = "k_im_pr2_sweep"
    else:
        n_launch = n_top
        algo = STAGE_BYTES_PER_UPDATE.get(top, 32) * nc * nv
        kname = top
    avg_s = t_top / n_launch * 1e-3
    stage_bw = algo / avg_s / 1e9
    # the pseudo-step as the unit: 240 B of compulsory FP64 traffic per cell*velocity (evolution and
    # residual, forward and backward wavefronts, update, accepted-state re-evaluation) at the
    # device-resident pseudo-step rate
    achieved = BYTES_PER_UPDATE_PSEUDO_STEP * value / 1e9
    roofline = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "traffic": TRAFFIC_PER_PSEUDO_STEP_8X64X1024 if (case.nx, case.ny, nv) == (8, 64, 1024) else None,
                "traffic_source": "ncu launch list, cold-cache sum over one pseudo-step's launches",
                "kernel": "ImplicitSteady pseudo-step (one CUDA graph node group, 16 launches: the PR(2) "
                          "sweeps share one)",
                "bytes_per_update": BYTES_PER_UPDATE_PSEUDO_STEP, "peak_source": peak_kind,
                "pseudo_step_us": ms / args.steps / (sum(pseudo) / len(pseudo)) * 1e3,
                "dominant_stage": {"stage": top, "kernel": kname, "avg_us_per_launch": avg_s * 1e6,
                                   "algorithmic_bytes_per_launch": algo, "achieved_gbs": stage_bw,
                                   "frac": stage_bw / peak},
                "stage_share": {k: t / stot for k, (t, _) in stimes.items()},
                "stage_us_per_pseudo_step": {k: 1e3 * t / max(n, 1) for k, (t, n) in stimes.items()},
                "stage_us_ungraphed": {k: 1e3 * t / max(n, 1) for k, (t, n) in ustimes.items()},
                "note": "one 8.4 MB instance is L2-resident and the step is latency-bound: pr2_sweep and "
                        "the LU-SGS stages are Gauss-Seidel wavefronts, chains of (rows+nx-1) dependent "
                        "relaxations per pass; stage times come from events captured into the batch graphs "
                        "(the last pseudo-step of each of %d batches); stage_us_ungraphed: the same stages "
                        "launched one by one, launch gaps included" % (GRAPH_PROFILE_STEPS // 8)}
    fpk = fp64_peak(f"cuda:{local}")
    roofline["fp64"] = fp64_fraction(FLOPS_PER_UPDATE["implicit_steady"], value / world, fpk)

    # ---------------- the 1e-10 residual tolerance of the headline metric (the reference's case file uses 1e-8)
    s10 = Solver(case.with_(residual_tol=1e-10), *vel, device=local)
    s10.init_freestream()
    s10.implicit_init()
    t10 = time.perf_counter()
    d10, c10, r10 = s10.step_implicit(TOL10_MAX_PSEUDO_STEPS)
    t10 = time.perf_counter() - t10
    s10.close()
    tol10 = {"converged": bool(c10), "pseudo_steps": int(d10), "wall_s": t10,
             "science_1_4": [float(x) for x in r10[12:16]], "Rh_Rb": [float(r10[24]), float(r10[25])],
             "note": "science_3 (the rho V residual relative to a near-zero reference) decays slowly below "
                     "1e-8 (9.8e-9 at 1100 pseudo-steps, 1.7e-9 at 3000); the reference's case file stops at 1e-8"}

    # ---------------- the plain explicit step, for context (config: CFL 0.5, omega 0.81, 1000 steps)
    se = Solver(baseline_explicit_case(), *vel, device=local)
    se.init_freestream()
    se.step_explicit(EXPLICIT_STEPS)
    se.init_freestream()
    sx = torch.cuda.ExternalStream(se.stream)
    x0, x1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(sx):
        x0.record(sx)
        se.step_explicit(EXPLICIT_STEPS)
        x1.record(sx)
    x1.synchronize()
    xms = x0.elapsed_time(x1)
    se.profile(True)
    se.step_explicit(100)
    kt = {k: se.profile_read(k) for k in ("slopes", "faces", "walls", "cells")}
    se.profile(False)
    se.close()
    explicit = {"value": nc * nv * EXPLICIT_STEPS / (xms * 1e-3), "unit": UNIT, "ms_per_solver_step": xms / EXPLICIT_STEPS,
                "config": "Explicit 8x64x1024, CFL 0.5, omega 0.81, 1000 steps from the cold start, CUDA graphs",
                "kernel_avg_us": {k: 1e3 * t / max(n, 1) for k, (t, n) in kt.items()},
                "faces_roofline_frac": (BYTES_PER_UPDATE_EXPLICIT * nc * nv / (kt["faces"][0] / kt["faces"][1] * 1e-3) / 1e9) / peak}
    explicit["fp64"] = fp64_reference_work(FLOPS_PER_UPDATE["explicit"], explicit["value"], fpk)

    # ---------------- HighOrderImplicit: the cold start to the 3000 pseudo-step cap (the reference run
    # also stops at its iteration limit, analysis.json high_implicit status)
    sh = Solver(reference_case("HighOrderImplicit"), *vel, device=local)
    sh.init_freestream()
    sh.implicit_init()
    sh.step_implicit(16)                      # graph capture and warm-up
    sh.init_freestream()
    sh.implicit_init()
    hstream = torch.cuda.ExternalStream(sh.stream)
    h0, h1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(hstream):
        h0.record(hstream)
        done_h, conv_h, rep_h = sh.step_implicit(HO_MAX_PSEUDO_STEPS)
        h1.record(hstream)
    h1.synchronize()
    hms = h0.elapsed_time(h1)
    ho_value = nc * nv * done_h / (hms * 1e-3)
    high_order = {"value": ho_value, "unit": UNIT, "pseudo_steps": int(done_h), "converged": bool(conv_h),
                  "wall_s": hms * 1e-3, "ms_per_pseudo_step": hms / max(done_h, 1),
                  "c_minus_1": float(rep_h[52]), "science_1_4": [float(x) for x in rep_h[12:16]],
                  "Rh_Rb": [float(rep_h[24]), float(rep_h[25])],
                  "hbm_roofline_frac": BYTES_PER_UPDATE_PSEUDO_STEP * ho_value / 1e9 / peak,
                  "fp64": fp64_reference_work(FLOPS_PER_UPDATE["high_order_implicit"], ho_value, fpk),
                  "config": "HighOrderImplicit 8x64x1024 (WENO5-AO S2 evolution, PR2 + LU-SGS, 8 slabs), CFL 0.1, "
                            "nCFL 1000, mass rescale on, cold start, 3000 pseudo-step cap; FP64-bound (the "
                            "closures and WENO templates), so the HBM fraction is small by construction"}
    sh.close()

    # ---------------- the refined HighOrderImplicit variant: 16x128 cells, 48x48 velocities
    from ugks2d_high_order_b200.case import refined_high_order_case, velocity_table
    rcase = refined_high_order_case()
    rtab = velocity_table(48)
    sr = Solver(rcase, *rtab, device=local)
    sr.init_freestream()
    sr.implicit_init()
    sr.step_implicit(8)
    rstream = torch.cuda.ExternalStream(sr.stream)
    r0, r1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(rstream):
        r0.record(rstream)
        done_r, _, rep_r = sr.step_implicit(REFINED_PSEUDO_STEPS)
        r1.record(rstream)
    r1.synchronize()
    rms = r0.elapsed_time(r1)
    sr.close()
    rcv = rcase.nx * rcase.ny * len(rtab[0])
    high_order["refined"] = {"value": rcv * done_r / (rms * 1e-3), "unit": UNIT, "pseudo_steps": int(done_r),
                             "ms_per_pseudo_step": rms / max(done_r, 1),
                             "cap_3000_estimate_s": 3000 * rms / max(done_r, 1) * 1e-3,
                             "c_minus_1": float(rep_r[52]),
                             "config": "HighOrderImplicit 16x128 cells, 48x48 velocities (generated half-range "
                                       "table, scale 2), 8 slabs; pseudo-steps 9-%d of the cold start"
                                       % (8 + REFINED_PSEUDO_STEPS)}

    # ---------------- S2CN2, the explicit high-order step
    sc = Solver(reference_case("S2CN2"), *vel, device=local)
    sc.init_freestream()
    sc.step_s2cn2(8)
    cstream = torch.cuda.ExternalStream(sc.stream)
    c0, c1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(cstream):
        c0.record(cstream)
        done_c2, rep_c2 = sc.step_s2cn2(S2CN2_STEPS)
        c1.record(cstream)
    c1.synchronize()
    cms = c0.elapsed_time(c1)
    sc.close()
    cn_value = nc * nv * done_c2 / (cms * 1e-3)
    s2cn2 = {"value": cn_value, "unit": UNIT, "steps": int(done_c2), "ms_per_step": cms / max(done_c2, 1),
             "cnres": float(rep_c2[1]), "mmerr": float(rep_c2[2]), "drift": float(rep_c2[9]),
             "hbm_roofline_frac": BYTES_PER_UPDATE_EXPLICIT * cn_value / 1e9 / peak,
             "fp64": fp64_reference_work(FLOPS_PER_UPDATE["s2cn2"], cn_value, fpk),
             "config": "S2CN2 8x64x1024, CFL 0.1, 8 steps warm-up then 400 steps, two steps per CUDA graph; "
                       "FP64-bound"}
    # the research wall variants of the same step (FluxWall_type 0; W1T; W1T + W1D; W2R at Pr 1)
    variants = {}
    for vname, fields in (("kinetic_wall", dict(flux_wall=0)),
                          ("w1t_midpoint", dict(flux_wall=0, s2w1_time_centered=1)),
                          ("w1d_face_time", dict(flux_wall=0, s2w1_time_centered=1, s2w1d_face_time=1)),
                          ("w2r_shared", dict(pr=1.0, s2w2r_shared_predictor=1))):
        sv = Solver(reference_case("S2CN2").with_(**fields), *vel, device=local)
        sv.init_freestream()
        sv.step_s2cn2(4)
        vstream = torch.cuda.ExternalStream(sv.stream)
        v0, v1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(vstream):
            v0.record(vstream)
            done_v, rep_v = sv.step_s2cn2(VARIANT_STEPS)
            v1.record(vstream)
        v1.synchronize()
        vms = v0.elapsed_time(v1) / max(done_v, 1)
        sv.close()
        variants[vname] = {"ms_per_step": vms, "vs_delivered_step": vms / s2cn2["ms_per_step"], "steps": int(done_v),
                           "value": nc * nv / (vms * 1e-3), "drift": float(rep_v[9]), "cnres": float(rep_v[1])}
    s2cn2["wall_variants"] = variants

    # ---------------- batched S2CN2: 256 instances of uneven sizes
    from ugks2d_high_order_b200.batch import Batch
    from ugks2d_high_order_b200.case import batched_cases, velocity_table
    from ugks2d_high_order_b200.shard import instance_cost, shard
    bcases_all = batched_cases()
    bcosts = [instance_cost(c, n * n) for c, n in bcases_all]
    bcases, _ = shard(bcases_all, bcosts, rank, world)     # this rank's LPT share (all of it at N=1)
    tables = {n: velocity_table(n) for n in (24, 32, 48)}
    bt = Batch([(c, tables[n]) for c, n in bcases], device=local, max_streams=32)
    bt.init_freestream()
    k_tuned, tune_ms = bt.tune(steps=2)
    bt.init_freestream()
    bt.run(2)
    bstream = torch.cuda.ExternalStream(bt.stream)
    b0, b1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    blaunch0 = bt.launch_count
    barrier()
    with torch.cuda.stream(bstream):
        b0.record(bstream)
        bdone, bst = bt.run(BATCH_STEPS)
        b1.record(bstream)
    b1.synchronize()
    barrier()
    bms = max_over_ranks(b0.elapsed_time(b1))
    bcv = sum(bcosts)                                       # all instances, all ranks
    b_flops = sum(cv * S2CN2_FLOPS_BY_TABLE[n] for cv, (_, n) in zip(bcosts, bcases_all))
    b_value = bcv * BATCH_STEPS / (bms * 1e-3)
    batched = {"value": b_value, "unit": UNIT, "instances": len(bcases_all), "instances_this_rank": len(bcases),
               "cell_velocities_per_step": int(bcv), "scaling": "strong" if world > 1 else None,
               "steps": BATCH_STEPS, "ms_per_batched_step": bms / BATCH_STEPS, "streams": int(k_tuned),
               "all_accepted": bool((bdone == BATCH_STEPS).all() and not bst.any()),
               "vs_plain_s2cn2": b_value / (world * s2cn2["value"]),
               "fp64": dict(fp64_reference_work(b_flops / bcv, b_value / world, fpk),
                            note="flops per update counted per velocity set (24^2: %.0f, 32^2: %.0f, 48^2: %.0f) "
                                 "and weighted by each instance's cell-velocities" %
                                 (S2CN2_FLOPS_BY_TABLE[24], S2CN2_FLOPS_BY_TABLE[32], S2CN2_FLOPS_BY_TABLE[48])),
               "gpu_launches": int(bt.launch_count - blaunch0),
               "full_run_estimate_s": 2000 * bms / BATCH_STEPS * 1e-3,
               "config": "256 S2CN2 instances, seed PCG64(20261203), CFL 0.1, omega 0.5, cold start; 2 steps "
                         "warm-up after the autotuner; each bench step advances every instance by one step "
                         "(the distribution's full run is 2000 steps)"}
    bt.close()

    # ---------------- the adjoint workload: gradients of the wall shear and heat flux with respect
    # to wall speed, wall temperature and the tau scale through the S2CN2 steps of 64 cases of the batched
    # distribution at 8x64 cells and 32^2 velocities, checkpoint every 50 steps.  ADJ_CASES of them are timed
    # over one full checkpoint segment: the plain forward, and the gradient (the checkpointed forward and the
    # reverse sweep with recompute), each on the case's own stream with CUDA events.
    c5_all = [(c.with_(ny=64, dy=1.0 / 64), 32) for c, _ in batched_cases(64)]
    c5, _ = shard(c5_all, [1] * len(c5_all), rank, world)
    seed = np.array([1.0, 1.0, 1.0, 1.0])
    grads = []
    fwd_list, fc_list, bw_list = [], [], []
    for case, nva in c5[:ADJ_CASES]:
        sv = Solver(case, *tables[nva], device=local)
        try:
            st_ = torch.cuda.ExternalStream(sv.stream)
            sv.init_freestream(tnative=2.0)
            sv.step_s2cn2(2)   # graph capture; then a full-size gradient reserves the adjoint's memory
            sv.init_freestream(tnative=2.0)
            sv.s2cn2_forward_checkpointed(ADJ_STEPS, every=ADJ_EVERY)
            sv.s2cn2_backward(seed)
            sv.init_freestream(tnative=2.0)
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(5)]
            with torch.cuda.stream(st_):
                ev[0].record(st_)
                sv.step_s2cn2(ADJ_STEPS)
                ev[1].record(st_)
            ev[1].synchronize()
            sv.init_freestream(tnative=2.0)
            with torch.cuda.stream(st_):
                ev[2].record(st_)
                sv.s2cn2_forward_checkpointed(ADJ_STEPS, every=ADJ_EVERY)
                ev[3].record(st_)
                g = sv.s2cn2_backward(seed)
                ev[4].record(st_)
            ev[4].synchronize()
            fwd_list.append(ev[0].elapsed_time(ev[1]))
            fc_list.append(ev[2].elapsed_time(ev[3]))
            bw_list.append(ev[3].elapsed_time(ev[4]))
            grads.append([float(x) for x in g])
        finally:
            sv.close()
    # a run of several segments (all but the last recomputed from their checkpoints in the backward)
    long_fwd = long_grad = 0.0
    if c5:
        case, nva = c5[0]
        sv = Solver(case, *tables[nva], device=local)
        try:
            st_ = torch.cuda.ExternalStream(sv.stream)
            sv.init_freestream(tnative=2.0)
            sv.step_s2cn2(2)   # graph capture; then an untimed full-length gradient reserves its memory
            sv.init_freestream(tnative=2.0)
            sv.s2cn2_forward_checkpointed(ADJ_LONG_STEPS, every=ADJ_EVERY)
            sv.s2cn2_backward(seed)
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
            sv.init_freestream(tnative=2.0)
            with torch.cuda.stream(st_):
                ev[0].record(st_)
                sv.step_s2cn2(ADJ_LONG_STEPS)
                ev[1].record(st_)
            ev[1].synchronize()
            sv.init_freestream(tnative=2.0)
            with torch.cuda.stream(st_):
                ev[2].record(st_)
                sv.s2cn2_forward_checkpointed(ADJ_LONG_STEPS, every=ADJ_EVERY)
                sv.s2cn2_backward(seed)
                ev[3].record(st_)
            ev[3].synchronize()
            long_fwd, long_grad = ev[0].elapsed_time(ev[1]), ev[2].elapsed_time(ev[3])
        finally:
            sv.close()
    fwd_ms, fc_ms, bw_ms = sum(fwd_list), sum(fc_list), sum(bw_list)
    barrier()
    fwd_ms, fc_ms, bw_ms = max_over_ranks(fwd_ms), max_over_ranks(fc_ms), max_over_ranks(bw_ms)
    long_fwd, long_grad = max_over_ranks(long_fwd), max_over_ranks(long_grad)
    n_t = len(fwd_list)
    long_cost = long_grad / long_fwd if long_fwd > 0 else None
    adjoint = {"gradients": "hand-written discrete adjoint of the S2CN2 step (ugks_s2cn2_forward_checkpointed + "
                            "ugks_s2cn2_backward: checkpoint every %d steps; the backward recomputes each segment "
                            "from its checkpoint once, every step leaving the record its transpose reads, except "
                            "the last segment, whose states and records the forward leaves)" % ADJ_EVERY,
               "cases": len(c5_all), "cases_timed": n_t, "steps": ADJ_STEPS,
               "forward_ms_per_step": fwd_ms / (n_t * ADJ_STEPS),
               "checkpointed_forward_ms_per_step": fc_ms / (n_t * ADJ_STEPS),
               "backward_ms_per_step": bw_ms / (n_t * ADJ_STEPS),
               "gradient_ms_per_step": (fc_ms + bw_ms) / (n_t * ADJ_STEPS),
               "cost_vs_forward": (fc_ms + bw_ms) / fwd_ms,
               "backward_vs_forward": bw_ms / fwd_ms,
               "long_run": {"steps": ADJ_LONG_STEPS, "every": ADJ_EVERY, "forward_ms": long_fwd,
                            "gradient_ms": long_grad, "cost_vs_forward": long_cost,
                            "note": "the first case; all segments but the last are recomputed in the backward"},
               "full_run_estimate_s": (2000 * len(c5_all) * long_grad / ADJ_LONG_STEPS * 1e-3) if long_fwd > 0 else None,
               "grad_first_case": grads[0] if grads else None,
               "config": "%d of the 64 cases of the batched distribution at 8x64 cells, 32x32 velocities, from the "
                         "cold start; one checkpoint segment of %d steps each (cost_vs_forward); seed = sum of the "
                         "four wall outputs; every case runs on its own context and stream; long_run: %d steps of "
                         "the first case, the config's 2000-step run estimated from it" % (n_t, ADJ_STEPS, ADJ_LONG_STEPS)}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            cpu = cpu_baseline(case, vel)
            cpu["time_to_steady_estimate_s"] = cpu["seconds_per_pseudo_step"] * (sum(pseudo) / len(pseudo))
        except Exception as e:   # the oracle sample is optional for the device number
            cpu = {"value": None, "unit": UNIT, "cores": 0, "kind": "port", "sample": f"unavailable: {e}"}
        try:
            high_order["cpu_baseline"] = cpu_sample_high_order(vel)
            s2cn2["cpu_baseline"] = cpu_sample_s2cn2(vel)
        except Exception as e:
            high_order["cpu_baseline"] = s2cn2["cpu_baseline"] = {"value": None, "sample": f"unavailable: {e}"}

    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
                "time_to_steady_s": ms / args.steps * 1e-3,
                "pseudo_steps_to_gate": pseudo,
                "solve_ms": solve_ms,
                "config": {"workload": WORKLOAD, "updates_per_pseudo_step": nc * nv,
                           "parallelism": f"replicas x{world}" if world > 1 else "single instance",
                           "l2": "flushed (256 MB write) between bench steps; the 8.4 MB state is L2-resident within a solve"},
                "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": state_bytes,
                        "d2h_bytes_per_step": state_bytes, "time_to_steady_s": ems / args.steps * 1e-3},
                "gpu_launches": int(launches),
                "roofline": roofline,
                "cpu_baseline": cpu,
                "explicit_plain": explicit,
                "tol_1e-10": tol10,
                "high_order_implicit": high_order,
                "s2cn2": s2cn2,
                "batched": batched,
                "adjoint": adjoint,
                "clocks": clocks}
        print(json.dumps(line), flush=True)
    s.close()
    if pg:
        pg.destroy_process_group()


if __name__ == "__main__":
    main()
