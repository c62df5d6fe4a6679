#!/usr/bin/env python
"""Throughput of the 2D Rayleigh-Benard IMEX timestep on B200 (steps/s).

Workload (default): ChannelDomain(1024, 256; Lx=4, Lz=1), Boussinesq with tau/lift
boundary conditions, Ra=1e8, Pr=1, RK443, dt=0.01, Float64, seeded initial noise
1e-3 z(Lz-z) (the 1024x256 Rayleigh-Benard configuration of the benchmark plan).
One "step" is one timestep of that problem; the step is a CUDA graph replayed by
the library.  With N GPUs each rank runs an independent replica (the 2D path has
no cross-GPU exchange), the timed region is bracketed by barriers and the
device time is the max over ranks.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Prints one JSON line (rank 0).  `--impl reference` times the CPU restatement of
the reference's algorithm (oracle/, NumPy + SciPy SuperLU, all host threads) on the
same workload.
"""
from __future__ import annotations

import os as _os

# More hardware work queues than the default 8, so that the ensemble runner's
# worker streams really run side by side (read once, at CUDA initialisation).
_os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")
import argparse
import json
import math
import os
import statistics
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=None)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--scheme", choices=["RK443", "RK222", "SBDF2"], default="RK443")
    ap.add_argument("--config", choices=["c2", "c1"], default="c2")
    ap.add_argument("--e2e-steps", type=int, default=20)
    ap.add_argument("--tau-parts", type=int, default=0, choices=[0, 1, 4, 8, 16],
                    help="tau-solve partitions of the headline plan (0: chosen by the plan's tuner)")
    ap.add_argument("--precision", choices=["f64", "mixed"], default="f64",
                    help="arithmetic of the headline plan (mixed: FP32 transforms and products, FP64 tau LU)")
    ap.add_argument("--tensor-cores", action="store_true",
                    help="mixed headline plan: transform GEMMs on the tcgen05 tensor cores (TF32)")
    ap.add_argument("--x-form", type=int, default=0, choices=[0, 1, 2, 3],
                    help="x-products kernel of the headline plan: 1 per field, 2 batched (0: the tuner's choice; "
                         "with --tau-parts the plan's default, 1)")
    ap.add_argument("--cpu-steps", type=int, default=10,
                    help="timed steps of the CPU baseline leg (about 1 s each on 16 host threads)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--workload", choices=["rbc", "ensemble", "serving", "turb", "rbc3d"], default="rbc",
                    help="rbc: the single-instance step (headline); ensemble / serving: that workload alone")
    ap.add_argument("--no-ensemble", action="store_true", help="skip the ensemble summary in the rbc line")
    ap.add_argument("--no-serving", action="store_true", help="skip the serving summary in the rbc line")
    ap.add_argument("--no-mixed", action="store_true", help="skip the mixed-precision summary in the rbc line")
    ap.add_argument("--no-rbc3d", action="store_true", help="skip the 3D (256x256x128) summary in the rbc line")
    ap.add_argument("--rbc3d-grid", default="256x256x128", help="Nx x Ny x Nz of the 3D workload")
    ap.add_argument("--rbc3d-gemm", choices=["auto", "simt", "tensor"], default="auto",
                    help="3D z-transform GEMMs: the tuner's choice, SIMT FP32 or the streaming tcgen05 TF32x3 kernel")
    ap.add_argument("--rbc3d-quick", action="store_true",
                    help="3D workload without the FP64 comparison and the end-to-end run (profiling)")
    ap.add_argument("--serve-requests", type=int, default=60)
    ap.add_argument("--serve-budget-gb", type=float, default=40.0)
    ap.add_argument("--turb-n", type=int, default=1024)
    ap.add_argument("--ensemble-size", type=int, default=64)
    ap.add_argument("--ensemble-steps", type=int, default=100)
    return ap.parse_args()


# ---------------------------------------------------------------------------
# distributed plumbing (replicas only; used for the barrier and the max)
# ---------------------------------------------------------------------------
class Dist:
    def __init__(self, collectives: bool = True):
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local = int(os.environ.get("LOCAL_RANK", "0"))
        self.pg = None
        self.backend = None
        if self.world > 1 and collectives:
            import datetime

            import torch
            import torch.distributed as dist

            self.backend = os.environ.get("TB_DIST_BACKEND", "nccl")
            if self.backend == "nccl":
                torch.cuda.set_device(self.local)
                dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                        device_id=torch.device("cuda", self.local))
            else:
                dist.init_process_group(self.backend, timeout=datetime.timedelta(seconds=120))
            self.pg = dist

    def barrier(self):
        if self.pg:
            self.pg.barrier()

    def max(self, v: float) -> float:
        if not self.pg:
            return v
        import torch

        dev = "cuda" if self.backend == "nccl" else "cpu"
        t = torch.tensor([v], dtype=torch.float64, device=dev)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def gather(self, obj):
        """Every rank's obj, in rank order (host objects; statistics only)."""
        if not self.pg:
            return [obj]
        out = [None] * self.world
        self.pg.all_gather_object(out, obj)
        return out

    def close(self):
        if self.pg:
            self.pg.barrier()
            self.pg.destroy_process_group()


# ---------------------------------------------------------------------------
# clock sampling during the timed region (NVML)
# ---------------------------------------------------------------------------
class ClockSampler:
    REASONS = {
        "gpu_idle": 0x1,
        "applications_clocks_setting": 0x2,
        "sw_power_cap": 0x4,
        "hw_slowdown": 0x8,
        "sync_boost": 0x10,
        "sw_thermal_slowdown": 0x20,
        "hw_thermal_slowdown": 0x40,
        "hw_power_brake_slowdown": 0x80,
    }

    def __init__(self, device: int, period: float = 0.005):
        self.device, self.period = device, period
        self.samples, self.reasons = [], set()
        self._stop = threading.Event()
        self.ok = False
        try:
            import pynvml

            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(device)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM)
            self.ok = True
        except Exception:
            self.max_mhz = None

    def _run(self):
        nv = self.nv
        while not self._stop.is_set():
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM))
                r = nv.nvmlDeviceGetCurrentClocksEventReasons(self.h)
                for name, bit in self.REASONS.items():
                    if r & bit and name != "gpu_idle":
                        self.reasons.add(name)
            except Exception:
                pass
            time.sleep(self.period)

    def __enter__(self):
        if self.ok:
            self._t = threading.Thread(target=self._run, daemon=True)
            self._t.start()
        return self

    def __exit__(self, *a):
        if self.ok:
            self._stop.set()
            self._t.join()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": self.max_mhz, "reasons": sorted(self.reasons), "samples": 0}
        return {"sm_mhz": statistics.median(self.samples), "sm_max_mhz": self.max_mhz,
                "reasons": sorted(self.reasons), "samples": len(self.samples)}


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            d = json.load(f)
        return d, "measured"
    except Exception:
        return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0}, "fallback"


# ---------------------------------------------------------------------------
# per-kernel algorithmic work (bytes moved by the algorithm, or flops)
# ---------------------------------------------------------------------------
def kernel_work(name: str, cfg, scheme: str):
    """(kind, amount per launch) with kind 'bytes' or 'flops'."""
    nk = cfg.Nx // 2 + 1
    plane = cfg.Nz * nk * 16
    N = cfg.Nz
    nb = {0: 3, 1: 4}
    n = 2 * N  # band rows per parity class
    if name == "z_backward_gemm":
        # values and z-derivatives from the even/odd coefficient halves: per field
        # (H x Ke + H x Ko) x 2 multiply-adds per column, H = ceil(Nz/2)
        H = (N + 1) // 2
        return "flops", 2.0 * 2 * H * N * (2 * nk) * 3
    if name == "z_forward_gemm":
        H = (N + 1) // 2
        return "flops", 2.0 * N * H * (2 * nk) * 3
    if name == "x_fft_products":
        # reads 12 half planes (values, z-derivatives; even/odd) and writes 3 planes
        return "bytes", 9.0 * plane
    if name == "tau_solve":
        # the banded LU factors themselves (forward 9 + backward 18 doubles per band row,
        # class and mode: pivot, 4 multipliers, 4 border multipliers; 1/diag, 12 U
        # entries, 4 border entries, store target; rows padded to a multiple of 48)
        # + Schur inverses; rhs read (4 planes); unknowns written (4 planes + taus).
        # The partitioned solve's extra response records are not algorithmic bytes.
        npad = (n + 47) // 48 * 48
        groups = (nk + 3) // 4
        fac = groups * 4 * (npad * 2 * (9 + 18) * 8 + 2 * 16 * 8)
        return "bytes", fac + 4.0 * plane + 4.0 * plane + 7 * nk * 16
    if name == "stage_lincomb":
        return "bytes", None  # depends on the stage; reported only if dominant
    if name == "lx_finalize":
        return "bytes", (4 + 3 + 4) * plane
    if name == "rk_final":
        return "bytes", None
    if name == "mass_apply":
        return "bytes", (3 + 4) * plane
    return "bytes", None


REF_SAMPLE_S = 60.0  # timed seconds of the CPU reference leg
REF_WARM_S = 30.0  # warm-up seconds of the CPU reference leg beyond its first 3 steps


def host_threads() -> int:
    """Host cores this process may run on (the CPU legs use all of them)."""
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def host_info(threads: int) -> dict:
    """The host the CPU legs run on: CPU model, core count, thread settings,
    and whether the reference itself (Julia + the Tarang.jl sources) could run
    here instead of the restatement."""
    import shutil

    model = None
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    model = line.split(":", 1)[1].strip()
                    break
    except OSError:
        pass
    julia = shutil.which("julia")
    return {
        "cpu_model": model,
        "nproc": os.cpu_count(),
        "threads_used": threads,
        "thread_settings": {"pocketfft_workers": threads, "per_mode_pool_threads": threads,
                            **{k: os.environ.get(k) for k in ("OPENBLAS_NUM_THREADS", "OMP_NUM_THREADS",
                                                              "MKL_NUM_THREADS")}},
        "julia": julia,
        "reference_runnable": False,
        "why_restatement": ("julia found at " + julia + " but the Tarang.jl sources and their FFTW/SuiteSparse "
                            "dependencies are not installed on this host") if julia else
                           "no julia executable on this host (probed with shutil.which at run time)",
    }


# ---------------------------------------------------------------------------
def run_reference(args, cfg, scheme, dist):
    """CPU restatement of the reference's algorithm, timed on the host cores."""
    if dist.rank != 0:
        return
    from oracle.tarang_oracle import RBCParams, run_rbc, rbc_initial_b, RBC2D, set_threads

    threads = set_threads(host_threads())
    p = RBCParams(Nx=cfg.Nx, Nz=cfg.Nz, Lx=cfg.Lx, Lz=cfg.Lz, Ra=cfg.Ra, Pr=cfg.Pr)
    sim = RBC2D(p)
    sim.set_b_grid(rbc_initial_b(p, cfg.seed))
    # Bounded sample: each full step takes seconds on the host.  The warm-up
    # (its first step factors every mode's LHS) runs at least min(--warmup, 3)
    # steps and stops after REF_WARM_S seconds beyond those; the timed steps
    # stop at --steps or after REF_SAMPLE_S seconds, whichever comes first.
    nwarm = 0
    t0 = time.perf_counter()
    while nwarm < args.warmup:
        if nwarm >= 3 and time.perf_counter() - t0 > REF_WARM_S:
            break
        sim.step(cfg.dt, scheme)
        nwarm += 1
    t0 = time.perf_counter()
    nsteps = 0
    while nsteps < args.steps:
        sim.step(cfg.dt, scheme)
        nsteps += 1
        if time.perf_counter() - t0 > REF_SAMPLE_S:
            break
    el = time.perf_counter() - t0
    v = nsteps / el
    out = {
        "impl": "reference",
        "metric": f"RBC 2D steps/s ({cfg.Nx}x{cfg.Nz}, {scheme}, Float64)",
        "value": v,
        "unit": "steps/s",
        "n_gpus": 0,
        "steps": nsteps,
        "warmup": nwarm,
        "requested": {"steps": args.steps, "warmup": args.warmup},
        "ms_per_step": 1e3 / v,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f64",
        "data": "synthetic (seeded PCG64 noise)",
        "config": workload_config(cfg, scheme, args),
        "cpu_baseline": {
            "value": v,
            "unit": "steps/s",
            "cores": threads,
            "kind": "port",
            "sample": f"{nsteps} steps (of --steps {args.steps}, capped at {REF_SAMPLE_S:.0f} s) after {nwarm} "
                      "warm-up steps (the first factors the tau LHS) "
                      f"of the full {cfg.Nx}x{cfg.Nz} problem; NumPy/SciPy restatement (SuperLU per mode), "
                      f"{threads} host threads (pocketfft workers, per-mode solves on a thread pool)",
            "host": host_info(threads),
        },
        "e2e": {"value": v, "unit": "steps/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(out), flush=True)


def workload_config(cfg, scheme, args):
    return {
        "workload": f"2D Rayleigh-Benard {cfg.Nx}x{cfg.Nz} Float64 {scheme} dt={cfg.dt}",
        "Nx": cfg.Nx,
        "Nz": cfg.Nz,
        "Lx": cfg.Lx,
        "Lz": cfg.Lz,
        "Ra": cfg.Ra,
        "Pr": cfg.Pr,
        "dt": cfg.dt,
        "timestepper": scheme,
        "dealias": 1.5,
        "global_batch": 1 if args.gpus in (None, 1) else args.gpus,
        "parallelism": "replicas",
        "l2": "working set (state, stage vectors, tau factors ~0.2 GB) exceeds the 126 MB L2",
    }


def cpu_baseline(cfg, scheme, nsteps):
    from oracle.tarang_oracle import RBCParams, RBC2D, rbc_initial_b, set_threads

    threads = set_threads(host_threads())
    p = RBCParams(Nx=cfg.Nx, Nz=cfg.Nz, Lx=cfg.Lx, Lz=cfg.Lz, Ra=cfg.Ra, Pr=cfg.Pr)
    sim = RBC2D(p)
    sim.set_b_grid(rbc_initial_b(p, cfg.seed))
    for _ in range(3):  # warm-up; the first step does the per-mode sparse LU factorisation
        sim.step(cfg.dt, scheme)
    t0 = time.perf_counter()
    for _ in range(nsteps):
        sim.step(cfg.dt, scheme)
    el = time.perf_counter() - t0
    return {
        "value": nsteps / el,
        "unit": "steps/s",
        "cores": threads,
        "kind": "port",
        "sample": f"{nsteps} steps of the full {cfg.Nx}x{cfg.Nz} {scheme} problem after 3 warm-up steps; "
                  "NumPy/SciPy restatement of the reference CPU path (SuperLU per Fourier mode), "
                  f"{threads} host threads (pocketfft workers, per-mode solves on a thread pool)",
        "host": host_info(threads),
    }


def run_ours(args, cfg, scheme, dist):
    import numpy as np
    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W
    from tarang_b200._lib import TB_FIELD_B, TB_FIELD_P, TB_FIELD_TAU, TB_FIELD_UX, TB_FIELD_UZ

    dev = dist.local
    torch.cuda.set_device(dev)
    dom = tb.ChannelDomain(cfg.Nx, cfg.Nz, Lx=cfg.Lx, Lz=cfg.Lz, arch=tb.GPU(dev))
    ts = {"RK222": 0, "RK443": 1, "SBDF2": 3}[scheme]
    from tarang_b200._lib import TB_PREC_F64, TB_PREC_MIXED

    plan = tb.Plan(dom, cfg.kappa, cfg.nu, cfg.Lz, 0.0, ts,
                   precision=TB_PREC_MIXED if args.precision == "mixed" else TB_PREC_F64)
    if args.tensor_cores:
        plan.set_gemm_path(True)
    b0 = plan.forward(W.rbc_initial_grid(cfg))
    plan.set_state(TB_FIELD_B, b0)

    # warm-up (the first call factors the tau systems and captures the step graph),
    # then the plan's kernel shapes are tuned on a few steps (state restored)
    if args.tau_parts or args.x_form:
        plan.set_variant(tau_parts=args.tau_parts, xrows=args.x_form)
        if args.tau_parts and plan.solve_form():
            plan.set_solve_form(False)  # the partitions asked for, not the dense inverses
    plan.step(cfg.dt, args.warmup)
    tuned = plan.variant() if (args.tau_parts or args.x_form) else plan.tune(cfg.dt, trial_steps=3)
    if args.tensor_cores:
        plan.set_gemm_path(True)  # (the tuner picks a path of its own)
    plan.step(cfg.dt, 1)

    # timed region: K graph replays, device time from CUDA events on the plan's stream
    dist.barrier()
    torch.cuda.synchronize()
    with ClockSampler(dev) as clk:
        plan.step(cfg.dt, args.steps)
    torch.cuda.synchronize()
    dist.barrier()
    ms_local = plan.last_step_ms()
    ms = dist.max(ms_local)
    value = dist.world * args.steps / (ms / 1e3)
    kps = plan.kernels_per_step()

    # per-kernel breakdown (eager launches with CUDA events around each kernel)
    nprof = max(3, min(20, args.steps))
    plan.set_profiling(True)
    plan.step(cfg.dt, nprof)
    prof = plan.profile()
    plan.set_profiling(False)
    tot = sum(v[0] for v in prof.values())
    shares = {k: v[0] / tot for k, v in prof.items()}
    top = max(prof, key=lambda k: prof[k][0])
    peaks, peak_src = measured_peaks()
    kind, work = kernel_work(top, cfg, scheme)
    avg_ms = prof[top][0] / prof[top][1]
    roof = None
    if work is not None:
        if kind == "bytes":
            ach = work / (avg_ms / 1e3) / 1e9
            peak = peaks.get("hbm_gbs")
            roof = {"bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s", "frac": ach / peak,
                    "traffic": None, "kernel": top, "algorithmic_bytes_per_launch": work}
        else:
            ach = work / (avg_ms / 1e3) / 1e12
            peak = fp64_peak_tflops()
            roof = {"bound": "tensor", "achieved": ach, "peak": peak, "unit": "TFLOP/s",
                    "frac": ach / peak if peak else None, "traffic": None, "kernel": top,
                    "flops_per_launch": work, "peak_source": "cuBLAS FP64 GEMM (torch.matmul float64) measured in bench"}
        roof["avg_launch_ms"] = avg_ms
        roof["peak_source"] = roof.get("peak_source", f"MEASURED_PEAKS.json ({peak_src})")
    # DRAM traffic per launch (average over a step's launches of each kernel
    # name) from the committed ncu capture of this workload
    tpath = os.path.join(ROOT, "profiles", f"traffic_{cfg.Nx}x{cfg.Nz}_{scheme.lower()}.json")
    tr, tr_launches = {}, 0
    if os.path.exists(tpath):
        with open(tpath) as f:
            cap = json.load(f)
        tr = {k: v for k, v in cap.items() if not k.startswith("_")}
        tr_launches = cap.get("_launches_per_step", 0)
    if roof is not None and top in tr:
        roof["traffic"] = tr[top]
        roof["traffic_source"] = tpath.replace(ROOT + os.sep, "")
    model = W.step_model_bytes(cfg, scheme)
    step_s = ms / args.steps / 1e3
    step_roof = {"bytes_per_step_model": model, "achieved_gbs": model / step_s / 1e9,
                 "peak_gbs": peaks.get("hbm_gbs")}
    step_roof["frac"] = step_roof["achieved_gbs"] / step_roof["peak_gbs"]
    if set(tr) == set(prof) and tr_launches * nprof == sum(v[1] for v in prof.values()):
        # what the step really moves: measured DRAM bytes of every kernel
        # launch of one step (ncu), over the device time of a step
        meas = sum(tr[k] * prof[k][1] / nprof for k in prof)
        step_roof["measured_dram_bytes_per_step"] = meas
        step_roof["measured_frac"] = meas / step_s / (step_roof["peak_gbs"] * 1e9)
        step_roof["measured_source"] = tpath.replace(ROOT + os.sep, "")

    # end to end through the C ABI with host buffers: per step, upload the
    # step's inputs from pinned host memory, one step, download the whole
    # state.  One pinned host buffer holds b, u_x, u_z, p and the taus back to
    # back (the device order), so each direction is one copy.  The inputs are
    # the prognostic fields b, u_x, u_z: p and the taus are outputs of the
    # step's tau solves (the IMEX tableaus never apply L to the step's initial
    # state, and M has no p or tau columns; tests/test_gpu_state_io.py checks
    # that they do not change the step), so only the first three planes go up.
    nk = cfg.Nx // 2 + 1
    pinned = torch.empty((4 * cfg.Nz + 7) * nk, dtype=torch.complex128, pin_memory=True).numpy()
    host = {f: pinned[f * cfg.Nz * nk:(f + 1) * cfg.Nz * nk].reshape(cfg.Nz, nk)
            for f in (TB_FIELD_B, TB_FIELD_UX, TB_FIELD_UZ, TB_FIELD_P)}
    host[TB_FIELD_TAU] = pinned[4 * cfg.Nz * nk:].reshape(7, nk)
    for f in host:
        host[f][...] = plan.get_state(f)
    ne = args.e2e_steps
    dist.barrier()
    t0 = time.perf_counter()
    inputs = {f: host[f] for f in (TB_FIELD_B, TB_FIELD_UX, TB_FIELD_UZ)}
    for _ in range(ne):
        plan.set_states(inputs, keep_history=True, wait=False)  # queued: the step queues behind it
        plan.step_async(cfg.dt, 1)  # the read-back below queues behind the step and waits for all three
        plan.get_states(host)
    e2e_el = dist.max(time.perf_counter() - t0)
    sbytes = W.state_bytes(cfg)
    ibytes = 16 * 3 * cfg.Nz * nk
    e2e = {"value": dist.world * ne / e2e_el, "unit": "steps/s", "h2d_bytes_per_step": ibytes,
           "d2h_bytes_per_step": sbytes, "steps": ne,
           "what": "per step: tb_set_states(TB_NO_WAIT) of the step's inputs b,ux,uz from one pinned host buffer "
                   "(one copy), tb_step_async(1), tb_get_states of all fields (b,ux,uz,p,taus) back into it (one copy); "
                   "all three queued in order on the plan's stream, one host wait per step"}

    finite = all(np.isfinite(plan.get_state(f)).all() for f in (TB_FIELD_B, TB_FIELD_UZ))
    cpu = None
    if dist.rank == 0 and dist.world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline(cfg, scheme, args.cpu_steps)
    if dist.rank == 0:
        out = {
            "metric": f"RBC 2D steps/s ({cfg.Nx}x{cfg.Nz}, {scheme}, "
                      f"{'Float64' if args.precision == 'f64' else 'FP32 transforms + FP64 tau LU'})",
            "value": value,
            "unit": "steps/s",
            "n_gpus": dist.world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": ms / args.steps,
            "higher_is_better": True,
            "scaling": "weak",
            "vs_baseline": None,
            "dtype": "f64",
            "data": "synthetic (seeded PCG64 noise, the benchmark configuration's initial condition)",
            "config": workload_config(cfg, scheme, args),
            "clocks": clk.summary(),
            "e2e": e2e,
            "gpu_launches": kps * args.steps,
            "kernels_per_step": kps,
            "tuned": {"tau_solve_partitions": tuned[0], "x_products_form": tuned[1]},
            "roofline": roof,
            "step_roofline": step_roof,
            "kernel_shares": {k: round(v, 4) for k, v in sorted(shares.items(), key=lambda x: -x[1])},
            "kernel_avg_ms": {k: prof[k][0] / prof[k][1] for k in prof},
            "cpu_baseline": cpu,
            "finite": bool(finite),
        }

        if dist.world == 1 and not args.no_mixed:
            try:
                out["mixed"] = run_mixed(args, cfg, scheme, dev)
            except Exception as exc:  # reported, never fatal to the headline line
                out["mixed"] = {"error": f"{type(exc).__name__}: {exc}"}
        if dist.world == 1 and not args.no_mixed:
            try:
                out["c1"] = run_c1(args, dev)
            except Exception as exc:  # reported, never fatal to the headline line
                out["c1"] = {"error": f"{type(exc).__name__}: {exc}"}
        if dist.world == 1 and not args.no_mixed and scheme != "SBDF2":
            try:
                out["sbdf2"] = run_sbdf2(args, cfg, dev)
            except Exception as exc:  # reported, never fatal to the headline line
                out["sbdf2"] = {"error": f"{type(exc).__name__}: {exc}"}
        if dist.world == 1 and not args.no_rbc3d:
            try:
                out["rbc3d"] = run_rbc3d(args, dev)
            except Exception as exc:  # reported, never fatal to the headline line
                out["rbc3d"] = {"error": f"{type(exc).__name__}: {exc}"}
        if dist.world == 1 and not args.no_mixed:
            try:
                out["dense_lu"] = run_dense_lu(dev)
            except Exception as exc:  # reported, never fatal to the headline line
                out["dense_lu"] = {"error": f"{type(exc).__name__}: {exc}"}
    # sharded across every rank (collective statistics: all ranks take part)
    if not args.no_ensemble:
        try:
            ens_out = run_ensemble(args, dev, dist, keep_states=True)
        except Exception as exc:  # reported, never fatal to the headline line
            ens_out = {"error": f"{type(exc).__name__}: {exc}"}
        try:
            ens_mixed = run_ensemble(args, dev, dist, mixed=True, keep_states=True)
            f64s, mxs = ens_out.pop("final_states", None), ens_mixed.pop("final_states", None)
            if f64s and mxs:
                import numpy as np

                ens_mixed["max_rel_l2_vs_f64_members"] = float(max(
                    np.linalg.norm(m[i] - f[i]) / np.linalg.norm(f[i]) for m, f in zip(mxs, f64s) for i in (0, 1)))
            if "plain_gpu" in ens_out:
                ens_mixed["speedup_vs_f64_plain_gpu"] = ens_mixed["value"] / ens_out["plain_gpu"]["value"]
            ens_out["mixed"] = ens_mixed
        except Exception as exc:  # reported, never fatal to the headline line
            ens_out["mixed"] = {"error": f"{type(exc).__name__}: {exc}"}
        ens_out.pop("final_states", None)
    if not args.no_serving:
        try:
            srv_out = run_serving(args, dev, dist)
        except Exception as exc:  # reported, never fatal to the headline line
            srv_out = {"error": f"{type(exc).__name__}: {exc}"}
    if dist.rank == 0:
        if not args.no_ensemble:
            out["ensemble"] = ens_out
        if not args.no_serving:
            out["serving"] = srv_out
        out["summary"] = summarize(out)  # last key: compact, so a truncated tail still carries it
        print(json.dumps(out), flush=True)


def summarize(out: dict) -> dict:
    """The headline and every secondary workload's main numbers, rounded."""

    def g(d, *keys):
        for k in keys:
            if not isinstance(d, dict) or k not in d or d[k] is None:
                return None
            d = d[k]
        if isinstance(d, float):  # 4 decimals, or 3 significant digits for small values (errors)
            return float(f"{d:.3g}") if 0.0 < abs(d) < 1e-2 else round(d, 4)
        return d

    s = {"steps_per_s": g(out, "value"), "e2e_steps_per_s": g(out, "e2e", "value"),
         "tau_solve_frac": g(out, "roofline", "frac"), "step_model_frac": g(out, "step_roofline", "frac"),
         "step_measured_frac": g(out, "step_roofline", "measured_frac")}
    if "mixed" in out:
        errs = g(out, "mixed", "rel_l2_vs_f64_after_steps") or {}
        s["mixed"] = {"steps_per_s": g(out, "mixed", "value"), "max_rel_l2_vs_f64": max(errs.values()) if errs else None}
    if "c1" in out:
        s["c1_steps_per_s"] = g(out, "c1", "value")
    if "dense_lu" in out:
        s["dense_lu_ms"] = {"ours": g(out, "dense_lu", "ours_ms"), "vendor": g(out, "dense_lu", "vendor_ms")}
    if "sbdf2" in out:
        s["sbdf2"] = {"f64": g(out, "sbdf2", "f64", "value"), "mixed": g(out, "sbdf2", "mixed", "value")}
    if "rbc3d" in out:
        s["rbc3d"] = {"mixed": g(out, "rbc3d", "value"), "f64": g(out, "rbc3d", "f64_plan_steps_per_s")}
    if "ensemble" in out:
        s["ensemble"] = {"fused": g(out, "ensemble", "value"),
                         "per_member_streams": g(out, "ensemble", "per_member_streams", "value"),
                         "plain_gpu": g(out, "ensemble", "plain_gpu", "value"),
                         "mixed": g(out, "ensemble", "mixed", "value"),
                         "mixed_vs_f64_plain": g(out, "ensemble", "mixed", "speedup_vs_f64_plain_gpu"),
                         "mixed_err": g(out, "ensemble", "mixed", "max_rel_l2_vs_f64_members")}
    if "serving" in out:
        s["serving"] = {"saturated": g(out, "serving", "saturated", "solves_per_s"),
                        "plain_saturated": g(out, "serving", "plain_gpu_saturated", "solves_per_s"),
                        "saturated_cohorts": g(out, "serving", "saturated_with_cohorts", "solves_per_s"),
                        "replay_p50_ms": g(out, "serving", "replay", "p50_ms"),
                        "replay_p99_ms": g(out, "serving", "replay", "p99_ms")}
    return s


def run_ensemble(args, dev, dist=None, mixed=False, keep_states=False):
    """Batched ensemble (independent 2D RBC instances of uneven size, RK222):
    instance steps per second of the ensemble runner against the plain GPU form
    (the same plans stepped one after another), and time-to-solution p50/p99.
    Under N ranks the members are sharded by cost (shard_instances) with no
    data-path collective; only the statistics are gathered."""
    import numpy as np
    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W

    members = W.ensemble_members(args.ensemble_size)
    world = dist.world if dist else 1
    rank = dist.rank if dist else 0
    shards = W.shard_instances([W.instance_cost(c) for c in members], world)
    members = [members[i] for i in shards[rank]]
    from tarang_b200._lib import TB_PREC_F64, TB_PREC_MIXED

    prec = TB_PREC_MIXED if mixed else TB_PREC_F64
    plans, init = [], []
    for c in members:
        dom = tb.ChannelDomain(c.Nx, c.Nz, Lx=c.Lx, Lz=c.Lz, arch=tb.GPU(dev))
        plan = tb.Plan(dom, c.kappa, c.nu, c.Lz, 0.0, 0, precision=prec)
        b0 = plan.forward(W.rbc_initial_grid(c))
        plan.set_state(0, b0)
        plans.append(plan)
        init.append(b0)
    zeros = [np.zeros_like(b) for b in init]

    def reset():
        for p, b, zz in zip(plans, init, zeros):
            p.set_state(0, b)
            p.set_state(1, zz)
            p.set_state(2, zz)

    dts = [c.dt for c in members]
    n = args.ensemble_steps
    # plain GPU form: each instance alone, one after another (factors/graphs warmed first)
    for p, dt in zip(plans, dts):
        p.step(dt, 1)
    reset()
    torch.cuda.synchronize()
    done = []
    t0 = time.perf_counter()
    for p, dt in zip(plans, dts):
        p.step(dt, n)
        done.append((time.perf_counter() - t0) * 1e3)
    plain_s = time.perf_counter() - t0
    reset()
    ens = tb.Ensemble(plans)
    streams, gsteps = ens.tune(dts, trial_steps=8)
    tuned_parts = plans[0].variant()[0]
    tuned_fused, tuned_groups = ens.form()
    reset()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    ms, total = ens.run(dts, n)
    wall = time.perf_counter() - t0
    finite = all(np.isfinite(p.get_state(0)).all() for p in plans)
    # the stronger GPU comparator: every member its own plan, graphs launched
    # on the tuned worker streams (the ensemble runner's per-member form)
    stream_total = None
    if tuned_fused:
        ens.set_form(False)
        reset()
        torch.cuda.synchronize()
        _, stream_total = ens.run(dts, n)
        ens.set_form(True)
    part = {"steps": len(plans) * n, "total_ms": float(total), "ms": [float(v) for v in ms], "plain_s": plain_s,
            "plain_done_ms": done, "finite": bool(finite),
            "streams_total_ms": None if stream_total is None else float(stream_total)}
    final = [(p.get_state(0), p.get_state(2)) for p in plans] if keep_states else None
    parts = dist.gather(part) if dist else [part]
    agg = W.combine_ensemble(parts)
    sizes = {}
    for c in W.ensemble_members(args.ensemble_size):
        sizes[f"{c.Nx}x{c.Nz}"] = sizes.get(f"{c.Nx}x{c.Nz}", 0) + 1
    return {
        "metric": "ensemble instance steps/s",
        "value": agg["value"],
        "unit": "instance-steps/s",
        "members": agg["members"],
        "steps_each": n,
        "sizes": sizes,
        "n_gpus": world,
        "sharding": "members assigned to ranks by cost (longest processing time first), no collective"
                    if world > 1 else "one GPU",
        "scheme": "RK222",
        "dtype": "f32 transforms/products, f64 tau LU" if mixed else "f64",
        "final_states": final,
        "tuned": {"worker_streams": streams, "steps_per_graph": gsteps, "tau_solve_partitions": tuned_parts,
                  "fused_form": tuned_fused, "stacked_group_plans": tuned_groups},
        "time_to_solution_ms": {"p50": agg["p50_ms"], "p99": agg["p99_ms"], "max": agg["total_ms"]},
        "wall_s": wall,
        "plain_gpu": {"value": agg["plain_value"], "unit": "instance-steps/s",
                      "what": "the same plans stepped one after another with tb_step (host wall clock)",
                      "time_to_solution_ms": {"p50": agg["plain_p50_ms"], "p99": agg["plain_p99_ms"]}},
        "speedup_vs_plain_gpu": agg["value"] / agg["plain_value"],
        "per_member_streams": None if any(p["streams_total_ms"] is None for p in parts) else {
            "value": sum(p["steps"] for p in parts) / (max(p["streams_total_ms"] for p in parts) / 1e3),
            "unit": "instance-steps/s",
            "what": "the same members as separate plans, step graphs launched on the tuned worker streams "
                    "(device clock)"},
        "finite": all(p["finite"] for p in parts),
        "data": "synthetic: sizes, Ra, Pr and noise seeded (ensemble seed 7, member noise seed 1000+k)",
    }


def run_mixed(args, cfg, scheme, dev):
    """Mixed precision on the headline configuration: FP32 transforms and
    products, FP64 tau LU, solves and stage algebra.  Steps/s (CUDA-graph
    replay, device clock) and the relative L2 error of b, u_x, u_z after the
    same number of steps against the Float64 form (which tracks the CPU oracle
    to 1e-10)."""
    import numpy as np
    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W
    from tarang_b200._lib import TB_PREC_MIXED

    ts = {"RK222": 0, "RK443": 1, "SBDF2": 3}[scheme]
    dom = tb.ChannelDomain(cfg.Nx, cfg.Nz, Lx=cfg.Lx, Lz=cfg.Lz, arch=tb.GPU(dev))
    mixed = tb.Plan(dom, cfg.kappa, cfg.nu, cfg.Lz, 0.0, ts, precision=TB_PREC_MIXED)
    full = tb.Plan(dom, cfg.kappa, cfg.nu, cfg.Lz, 0.0, ts)
    b0 = full.forward(W.rbc_initial_grid(cfg))
    for pl in (mixed, full):
        pl.set_state(0, b0)
    n = args.steps
    mixed.step(cfg.dt, n)
    full.step(cfg.dt, n)
    err = {name: float(np.linalg.norm(mixed.get_state(f) - full.get_state(f)) / np.linalg.norm(full.get_state(f)))
           for f, name in ((0, "b"), (1, "ux"), (2, "uz"))}
    # timing: graph replay after warm-up, from the state reached above, with
    # the kernel shapes the plan's tuner picks (state restored by the tuner)
    tuned = mixed.tune(cfg.dt, trial_steps=3)
    mixed.step(cfg.dt, args.warmup)
    torch.cuda.synchronize()
    mixed.step(cfg.dt, n)
    ms = mixed.last_step_ms()
    return {
        "metric": f"RBC 2D steps/s ({cfg.Nx}x{cfg.Nz}, {scheme}, FP32 transforms/products + FP64 tau LU)",
        "value": n / (ms / 1e3),
        "unit": "steps/s",
        "ms_per_step": ms / n,
        "rel_l2_vs_f64_after_steps": err,
        "steps": n,
        "tuned": {"tau_solve_partitions": tuned[0], "x_products_form": tuned[1],
                  "tensor_core_gemms": mixed.gemm_path()},
        "dtype": "f32 transforms/products, f64 solves/stage algebra",
    }


def run_sbdf2(args, cfg, dev):
    """SBDF2 on the headline grid (the multistep half of the 1024x256
    benchmark): Float64 and mixed steps/s on the device clock (graph replay
    after warm-up), the step byte model's HBM fraction, and the mixed form's
    relative L2 error against Float64 after the same steps."""
    import numpy as np
    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W
    from tarang_b200._lib import TB_PREC_MIXED, TB_SBDF2

    dom = tb.ChannelDomain(cfg.Nx, cfg.Nz, Lx=cfg.Lx, Lz=cfg.Lz, arch=tb.GPU(dev))
    full = tb.Plan(dom, cfg.kappa, cfg.nu, cfg.Lz, 0.0, TB_SBDF2)
    mixed = tb.Plan(dom, cfg.kappa, cfg.nu, cfg.Lz, 0.0, TB_SBDF2, precision=TB_PREC_MIXED)
    b0 = full.forward(W.rbc_initial_grid(cfg))
    n = args.steps
    for pl in (full, mixed):
        pl.set_state(0, b0)
        pl.step(cfg.dt, n)
    err = {nm: float(np.linalg.norm(mixed.get_state(f) - full.get_state(f)) / np.linalg.norm(full.get_state(f)))
           for f, nm in ((0, "b"), (1, "ux"), (2, "uz"))}
    peaks, _ = measured_peaks()
    model = W.step_model_bytes(cfg, "SBDF2")
    out = {}
    for name, pl in (("f64", full), ("mixed", mixed)):
        tuned = pl.tune(cfg.dt, trial_steps=3)
        pl.step(cfg.dt, args.warmup)
        torch.cuda.synchronize()
        pl.step(cfg.dt, n)
        ms = pl.last_step_ms() / n
        out[name] = {"value": 1e3 / ms, "ms_per_step": ms, "tuned": list(tuned),
                     "step_roofline_frac": model / (ms * 1e-3) / (peaks["hbm_gbs"] * 1e9)}
    return {
        "metric": f"RBC 2D steps/s ({cfg.Nx}x{cfg.Nz}, SBDF2)",
        "unit": "steps/s",
        "value": out["f64"]["value"],
        "f64": out["f64"],
        "mixed": out["mixed"],
        "mixed_rel_l2_vs_f64_after_steps": err,
        "bytes_per_step_model": model,
        "steps": n,
        "dtype": "f64; mixed: f32 transforms/products, f64 solves/stage algebra",
    }


def run_c1(args, dev):
    """The small configuration (256x64, RK222, dt 0.125, 100 steps, Float64;
    the reference's own CPU-runnable case): steps/s on the device clock over
    the 100 steps (graph replay after warm-up on a copy of the state) and the
    step byte model's HBM fraction."""
    import numpy as np
    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W

    c = W.C1
    dom = tb.ChannelDomain(c.Nx, c.Nz, Lx=c.Lx, Lz=c.Lz, arch=tb.GPU(dev))
    pl = tb.Plan(dom, c.kappa, c.nu, c.Lz, 0.0, 0)
    b0 = pl.forward(W.rbc_initial_grid(c))
    pl.set_state(0, b0)
    pl.step(c.dt, max(args.warmup, 3))
    tuned = pl.tune(c.dt, trial_steps=3)
    pl.set_state(0, b0)
    for f in (1, 2, 3):
        pl.set_state(f, np.zeros_like(b0))
    torch.cuda.synchronize()
    n = 100
    pl.step(c.dt, n)
    ms = pl.last_step_ms() / n
    peaks, _ = measured_peaks()
    model = W.step_model_bytes(c, "RK222")
    return {
        "metric": f"RBC 2D steps/s ({c.Nx}x{c.Nz}, RK222, Float64, dt={c.dt})",
        "value": 1e3 / ms,
        "unit": "steps/s",
        "ms_per_step": ms,
        "steps": n,
        "bytes_per_step_model": model,
        "step_roofline_frac": model / (ms * 1e-3) / (peaks["hbm_gbs"] * 1e9),
        "tuned": list(tuned),
        "note": "the working set (~0.01 GB) stays in the 126 MB L2, so the HBM fraction is not a bound here; "
                "the step is launch- and latency-bound",
    }


def run_dense_lu(dev, n: int = 263, batch: int = 129, reps: int = 5):
    """BatchedDenseLU at the small configuration's size (129 Fourier modes,
    n = 4 Nz + 7 = 263 at Nz = 64): the library's batched complex LU
    (tb_batched_lu_factor, the drop-in for batched_factor! whose CUDA method
    calls getrf strided-batched) against torch.linalg.lu_factor on the same
    slices (the vendor batched getrf), device time of the factorisation, and
    the relative residual of a solve with each."""
    import ctypes

    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    g = torch.Generator(device="cpu").manual_seed(3)
    A0 = (torch.randn(batch, n, n, dtype=torch.complex128, generator=g)
          + n * torch.eye(n, dtype=torch.complex128)).to(dev)
    b = torch.randn(batch, n, dtype=torch.complex128, generator=g).to(dev)
    ctx = tb.api._context(dev)

    def ours():
        A = A0.transpose(1, 2).contiguous()  # column-major slices
        piv = torch.empty(batch, n, dtype=torch.int32, device=dev)
        bad = ctypes.c_int(-1)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        st = tb.lib.tb_batched_lu_factor(ctx, n, batch, ctypes.c_void_p(A.data_ptr()), ctypes.c_void_p(piv.data_ptr()),
                                         ctypes.byref(bad))
        e1.record()
        torch.cuda.synchronize()
        assert st == 0, st
        return e0.elapsed_time(e1), A, piv

    def vendor():
        A = A0.clone()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        LU, pv = torch.linalg.lu_factor(A)
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1), LU, pv

    ours()
    vendor()
    t_ours = min(ours()[0] for _ in range(reps))
    t_vendor = min(vendor()[0] for _ in range(reps))
    _, A, piv = ours()
    x = b.clone().contiguous()
    st = tb.lib.tb_batched_lu_solve(ctx, n, batch, ctypes.c_void_p(A.data_ptr()), ctypes.c_void_p(piv.data_ptr()),
                                    ctypes.c_void_p(x.data_ptr()))
    assert st == 0, st
    res = float((torch.linalg.norm(torch.einsum("bij,bj->bi", A0, x) - b) / torch.linalg.norm(b)).item())
    _, LU, pv = vendor()
    xv = torch.linalg.lu_solve(LU, pv, b.unsqueeze(-1)).squeeze(-1)
    resv = float((torch.linalg.norm(torch.einsum("bij,bj->bi", A0, xv) - b) / torch.linalg.norm(b)).item())
    return {"what": f"batched complex LU factorisation, {batch} slices of {n} x {n}",
            "ours_ms": t_ours, "vendor_ms": t_vendor, "vendor": "torch.linalg.lu_factor (batched getrf)",
            "ours_rel_residual": res, "vendor_rel_residual": resv}


def kernel_work3(name: str, c, npad_main: int, npad_perp: int):
    """Algorithmic bytes per launch of the 3D step kernels (None: not modelled)."""
    nk = (c.Nx // 2 + 1) * c.Ny
    plane = c.Nz * nk * 16
    H = c.Nz // 2
    My = -(-3 * c.Ny // 2) + (-(-3 * c.Ny // 2)) % 2
    slab8 = c.Nz * (c.Nx // 2 + 1) * My * 8  # one FP32 [z][kx][y] array
    groups = (nk + 3) // 4
    if name == "tau_solve":
        # LU records (forward 9 + backward 18 doubles per band row, class and mode),
        # Schur inverses, rhs (4 planes) in, unknowns (4 planes + 7 tau rows) out
        return groups * 4 * (npad_main * 2 * 27 * 8 + 2 * 16 * 8) + 8.0 * plane + 7 * nk * 16
    if name == "tau_solve_perp":
        return groups * 4 * (npad_perp * 2 * 27 * 8 + 2 * 16 * 8) + 2.0 * plane + 2 * nk * 16
    if name == "rhs3_xpass":
        return 16.0 * slab8  # 12 factor arrays in, 4 product arrays out (FP32)
    if name == "rhs3_yinv":
        return 16.0 * H * nk * 8 + 12.0 * slab8
    if name == "rhs3_yfwd":
        return 4.0 * slab8 + 4.0 * c.Nz * nk * 8
    if name == "lx_finalize":
        return (5 + 4 + 5) * plane
    if name == "mass_apply":
        return (4 + 5) * plane
    return None


def cpu_baseline_3d(c, nz_sample: int = 16, mode_sample: int = 48):
    """CPU restatement on a bounded sample of the 3D workload, scaled to one
    RK222 step: one RHS evaluation on a z-slab with the full horizontal grid
    (scaled by Nz / nz_sample) and the per-mode sparse LU solve + L x product
    on a spread sample of Fourier modes (scaled to all modes)."""
    import numpy as np

    from oracle.tarang_oracle import RBC3D, RBC3Params, _pmap, rbc3_initial_b, set_threads

    threads = set_threads(host_threads())
    ps = RBC3Params(Nx=c.Nx, Ny=c.Ny, Nz=nz_sample, Lx=c.Lx, Ly=c.Ly, Lz=c.Lz, Ra=c.Ra, Pr=c.Pr)
    sim = RBC3D(ps)
    sim.set_b_grid(rbc3_initial_b(ps, c.seed, c.noise))
    rng = np.random.default_rng(0)
    u = [1e-3 * sim.b * rng.standard_normal() for _ in range(3)]
    t0 = time.perf_counter()
    sim.rhs(sim.b, *u)
    t_rhs = (time.perf_counter() - t0) * c.Nz / nz_sample
    pf = RBC3Params(Nx=c.Nx, Ny=c.Ny, Nz=c.Nz, Lx=c.Lx, Ly=c.Ly, Lz=c.Lz, Ra=c.Ra, Pr=c.Pr)
    simf = RBC3D(pf)
    nk = (c.Nx // 2 + 1) * c.Ny
    beta = c.dt * (1.0 - 1.0 / math.sqrt(2.0))
    nsample = max(mode_sample, 4 * threads)
    picks = [(int(i) % c.Ny, (int(i) // c.Ny) % (c.Nx // 2 + 1)) for i in np.linspace(0, nk - 1, nsample)]
    rhs = {m: rng.standard_normal(simf.mode_matrices(*m)[0].shape[0]) + 0j for m in picks}
    t0 = time.perf_counter()
    lus = dict(zip(picks, _pmap(lambda m: simf._lhs_lu(*m, 1.0, beta), picks)))
    t_fac = time.perf_counter() - t0

    def solve(m):
        x = lus[m].solve(rhs[m])
        return simf.mode_matrices(*m)[1] @ x

    t0 = time.perf_counter()
    _pmap(solve, picks)
    t_sol = time.perf_counter() - t0
    t_sol_all = t_sol * nk / nsample
    step_s = 2 * t_rhs + 2 * t_sol_all
    return {
        "value": 1.0 / step_s,
        "unit": "steps/s",
        "cores": threads,
        "kind": "port",
        "sample": f"one RHS evaluation on a {c.Nx}x{c.Ny}x{nz_sample} slab (scaled by {c.Nz}/{nz_sample}) and the "
                  f"per-mode SuperLU solve + L x of {nsample} of the {nk} Fourier modes at full n = "
                  f"{5 * c.Nz + 9} (scaled to all modes), combined for one RK222 step (2 RHS, 2 solve passes); "
                  f"the one-time factorisation ({t_fac * nk / nsample:.0f} s for all modes) is excluded; "
                  f"NumPy/SciPy restatement, {threads} host threads (pocketfft workers, per-mode solves "
                  "on a thread pool)",
        "rhs_s": t_rhs,
        "solves_s": t_sol_all,
    }


def run_rbc3d(args, dev, with_cpu=True):
    """3D Rayleigh-Benard 256x256x128, RK222, dt 5e-3, Ra 1e7, mixed precision
    (FP32 transforms and products, FP64 tau LU and solves), 50 steps captured
    as CUDA graphs.  Steps/s on the device clock, the error against the FP64
    plan (itself pinned to the oracle at 1e-10 on small grids), per-kernel
    shares, the end-to-end 50-step solve through the C ABI with host buffers."""
    import numpy as np
    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W
    from tarang_b200._lib import (TB_FIELD_B, TB_FIELD_P, TB_FIELD_UX, TB_FIELD_UY, TB_FIELD_UZ, TB_PREC_F64,
                                  TB_PREC_MIXED)

    nx, ny, nz = (int(v) for v in args.rbc3d_grid.lower().split("x"))
    c = W.RBC3Config(Nx=nx, Ny=ny, Nz=nz) if (nx, ny, nz) != (W.C3.Nx, W.C3.Ny, W.C3.Nz) else W.C3
    torch.cuda.set_device(dev)
    grid = W.rbc3_initial_grid(c)
    t0 = time.perf_counter()
    plan = tb.Plan3D(c.Nx, c.Ny, c.Nz, c.kappa, c.nu, 0, c.Lx, c.Ly, c.Lz, precision=TB_PREC_MIXED, device=dev)
    b0 = plan.forward(grid)
    plan.set_state(TB_FIELD_B, b0)
    plan.step(c.dt, 1)  # factors both tau systems for this dt and captures the step graph
    setup_s = time.perf_counter() - t0
    t1 = time.perf_counter()
    tuned = plan.tune(c.dt, trial_steps=3)  # kernel shapes (tau partitions, x-pass rows), state kept
    if args.rbc3d_gemm != "auto":
        plan.set_gemm_path(args.rbc3d_gemm == "tensor")
    tune_s = time.perf_counter() - t1
    plan.step(c.dt, max(args.warmup, 3))
    torch.cuda.synchronize()
    with ClockSampler(dev) as clk:
        plan.step(c.dt, c.steps)
    torch.cuda.synchronize()
    ms = plan.last_step_ms()
    value = c.steps / (ms / 1e3)
    kps = plan.kernels_per_step()
    plan.set_profiling(True)
    plan.step(c.dt, 3)
    prof = plan.profile()
    plan.set_profiling(False)
    tot = sum(v[0] for v in prof.values())
    peaks, peak_src = measured_peaks()
    npad_main = (2 * c.Nz + 3 + 47) // 48 * 48
    npad_perp = (c.Nz // 2 + 47) // 48 * 48
    kernels = {}
    for k, (t, n) in sorted(prof.items(), key=lambda x: -x[1][0]):
        e = {"share": round(t / tot, 4), "avg_ms": t / n, "launches_per_step": n / 3}
        w = kernel_work3(k, c, npad_main, npad_perp)
        if w is not None:
            e["algorithmic_GBs"] = w / (t / n / 1e3) / 1e9
            e["frac_of_hbm_peak"] = e["algorithmic_GBs"] / peaks["hbm_gbs"]
        kernels[k] = e
    top = max(prof, key=lambda k: prof[k][0])
    model = W.step_model_bytes3(c)
    nk = (c.Nx // 2 + 1) * c.Ny
    phi_ours = nk * 8.0 * (2 * npad_main * 27 + 2 * npad_perp * 27 + 4 * 16)
    step_roof = {"bytes_per_step_model": model, "achieved_gbs": model / (ms / c.steps / 1e3) / 1e9,
                 "peak_gbs": peaks["hbm_gbs"], "peak_source": f"MEASURED_PEAKS.json ({peak_src})",
                 "phi_nominal_bytes": nk * (5 * c.Nz + 9) * 848.0, "phi_built_bytes": phi_ours,
                 "note": "the byte model charges the nominal bordered-banded LHS (n x 848 B per mode) on 4 reads "
                         "per step; the built real banded factors are phi_built_bytes per read"}
    step_roof["frac"] = step_roof["achieved_gbs"] / step_roof["peak_gbs"]
    if args.rbc3d_quick:
        return {"metric": f"RBC 3D steps/s ({c.Nx}x{c.Ny}x{c.Nz}, {c.scheme}, mixed)", "value": value,
                "ms_per_step": ms / c.steps, "kernels": kernels, "step_roofline": step_roof, "tuned": tuned}
    # error against the FP64 plan from the same initial state
    for f in (TB_FIELD_UX, TB_FIELD_UY, TB_FIELD_UZ, TB_FIELD_P):
        plan.set_state(f, np.zeros((c.Nz, c.Ny, c.Nx // 2 + 1), np.complex128))
    plan.set_state(TB_FIELD_B, b0)
    full = tb.Plan3D(c.Nx, c.Ny, c.Nz, c.kappa, c.nu, 0, c.Lx, c.Ly, c.Lz, precision=TB_PREC_F64, device=dev)
    full.set_state(TB_FIELD_B, b0)
    plan.step(c.dt, c.steps)
    full.step(c.dt, c.steps)  # the first call at this dt also factors and captures the step graph
    err = {}
    for f, name in ((TB_FIELD_B, "b"), (TB_FIELD_UX, "ux"), (TB_FIELD_UY, "uy"), (TB_FIELD_UZ, "uz")):
        a, b = plan.get_state(f), full.get_state(f)
        err[name] = float(np.linalg.norm(a - b) / np.linalg.norm(b))
    finite = bool(np.isfinite(plan.get_state(TB_FIELD_UZ)).all())
    full.step(c.dt, c.steps)  # the FP64 plan's step rate, timed on its own graph replays
    ms64 = full.last_step_ms()
    del full
    # end to end: the 50-step solve through the C ABI with pinned host buffers
    shape = (c.Nz, c.Ny, c.Nx // 2 + 1)
    hin = {f: torch.zeros(shape, dtype=torch.complex128, pin_memory=True).numpy()
           for f in (TB_FIELD_B, TB_FIELD_UX, TB_FIELD_UY, TB_FIELD_UZ)}
    hin[TB_FIELD_B][...] = b0
    hout = {f: torch.empty(shape, dtype=torch.complex128, pin_memory=True).numpy()
            for f in (TB_FIELD_B, TB_FIELD_UX, TB_FIELD_UY, TB_FIELD_UZ, TB_FIELD_P)}
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for f, a in hin.items():
        plan.set_state(f, a)
    plan.step(c.dt, c.steps)
    for f, a in hout.items():
        tb.lib.tb_get_state(plan.ptr, f, a.ctypes.data_as(__import__("ctypes").c_void_p), 0)
    e2e_s = time.perf_counter() - t0
    fb = int(np.prod(shape)) * 16
    out = {
        "metric": f"RBC 3D steps/s ({c.Nx}x{c.Ny}x{c.Nz}, {c.scheme}, FP32 transforms/products + FP64 tau LU)",
        "value": value,
        "unit": "steps/s",
        "ms_per_step": ms / c.steps,
        "steps": c.steps,
        "dtype": "f32 transforms/products, f64 tau factors/solves/stage algebra",
        "config": {"workload": f"3D Rayleigh-Benard {c.Nx}x{c.Ny}x{c.Nz} RK222 dt={c.dt} Ra={c.Ra:g} Pr={c.Pr:g}",
                   "Lx": c.Lx, "Ly": c.Ly, "Lz": c.Lz, "modes": nk, "n_per_mode": 5 * c.Nz + 9,
                   "l2": "working set (~15 GB of factors and stage vectors) far exceeds the 126 MB L2"},
        "data": "synthetic: b0 = Lz - z + 1e-3 z (Lz - z) xi, xi ~ N(0,1) from PCG64(42), u = 0",
        "setup_s": setup_s,
        "tuned": {"tau_solve_partitions": tuned[0], "xpass_rows_per_cta": tuned[1],
                  "tensor_core_gemms": plan.gemm_path(), "tune_s": tune_s},
        "clocks": clk.summary(),
        "gpu_launches": kps * c.steps,
        "kernels_per_step": kps,
        "step_roofline": step_roof,
        "top_kernel": top,
        "kernels": kernels,
        "rel_l2_vs_f64_plan_after_steps": err,
        "f64_plan_steps_per_s": c.steps / (ms64 / 1e3),
        "e2e": {"value": c.steps / e2e_s, "unit": "steps/s", "h2d_bytes_per_step": 4 * fb / c.steps,
                "d2h_bytes_per_step": 5 * fb / c.steps,
                "what": "tb_set_state of b, u_x, u_y, u_z from pinned host memory, tb_step(50), tb_get_state "
                        "of b, u, p to host; bytes averaged over the 50 steps"},
        "device_bytes": plan.device_bytes(),
        "finite": finite,
    }
    if with_cpu and not args.no_cpu_baseline:
        out["cpu_baseline"] = cpu_baseline_3d(c)
    return out


def run_turb(args, dev):
    """One FP32 decaying-turbulence instance (N x N, DiagonalIMEX SBDF2,
    nu = 1e-4, dt = 2e-3, k^-3 initial spectrum): steps/s on the device clock."""
    import torch

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W

    N = args.turb_n
    t = tb.Turb2D(N, N, 1e-4, W.turb_initial_spec(N, 7000), device=dev)
    t.step(2e-3, args.warmup)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    t.step(2e-3, args.steps)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1)
    return {"metric": f"2D decaying turbulence steps/s ({N}x{N}, FP32, DiagonalIMEX SBDF2)",
            "value": args.steps / (ms / 1e3), "unit": "steps/s", "ms_per_step": ms / args.steps,
            "steps": args.steps, "warmup": args.warmup, "dtype": "f32",
            "data": "synthetic: k^-3 spectrum, random phases (seed 7000)"}


def run_serving(args, dev, dist=None):
    """Serving mix: seeded Poisson arrivals (20/s) of RBC channel runs and FP32
    decaying turbulence, 50-500 steps each, admitted by HBM budget.  Replayed
    through the request server (continuous batching) and through the plain GPU
    form (one request at a time); also the saturated throughput with every
    request queued at once.  Under N ranks the requests are sharded by cost
    (each rank serves its share at the original arrival times, no data-path
    collective) and the statistics are gathered."""
    import numpy as np

    from __graft_entry__ import load_package

    tb = load_package()
    from tarang_b200 import workloads as W

    reqs = W.serving_requests(args.serve_requests)
    world = dist.world if dist else 1
    rank = dist.rank if dist else 0
    mine = set(W.shard_instances([W.instance_cost(r) for r in reqs], world)[rank])
    prepared = []
    for k, r in enumerate(reqs):
        if k not in mine:
            prepared.append(None)
        elif r.kind == "rbc":
            c = r.rbc
            prepared.append((tb.rbc_desc(c.Nx, c.Nz, c.kappa, c.nu, 0, Lx=c.Lx, Lz=c.Lz), r.dt, r.nsteps,
                             W.rbc_initial_grid(c)))
        else:
            prepared.append((tb.turb_desc(r.N, r.N, r.nu), r.dt, r.nsteps, W.turb_initial_spec(r.N, r.seed)))
    budget = int(args.serve_budget_gb * (1 << 30))

    def replay(max_running, timed_arrivals, chunk=10, subset=None, cohort=1):
        subset = mine if subset is None else (subset & mine)
        srv = tb.Server(budget_bytes=budget, max_running=max_running, chunk_steps=chunk, device=dev)
        srv.set_cohort(cohort)
        t0 = time.perf_counter()
        ids, steps = [], 0
        for k, r in enumerate(reqs):
            if k not in subset:
                continue
            d, dt, n, init = prepared[k]
            if timed_arrivals:
                wait = r.arrival_s - (time.perf_counter() - t0)
                if wait > 0:
                    time.sleep(wait)
            ids.append(srv.submit(d, dt, n, init))
            steps += n
        srv.wait_all()
        wall = time.perf_counter() - t0
        st = srv.stats()
        polls = [srv.poll(i) for i in ids]
        ok = all(p[0] == tb._lib.TB_REQ_DONE for p in polls)
        srv.close()
        part = {"completed": int(st["completed"]), "steps": steps, "wall_s": wall,
                "tts_ms": [float(p[1]) for p in polls], "failed": int(st["failed"]), "all_done": ok,
                "peak_running": int(st["peak_running"]), "peak_bytes": int(st["peak_bytes"]),
                "mean_wait_ms": float(st["mean_wait_ms"]), "mean_setup_ms": float(st["mean_setup_ms"]),
                "peak_cohort": int(st["peak_cohort"]), "cohort_requests": int(st["cohort_requests"])}
        parts = dist.gather(part) if dist else [part]
        agg = W.combine_serving(parts)
        return {"solves_per_s": agg["solves_per_s"], "steps_per_s": agg["steps_per_s"], "p50_ms": agg["p50_ms"],
                "p99_ms": agg["p99_ms"], "mean_queue_wait_ms": float(np.mean([p["mean_wait_ms"] for p in parts])),
                "mean_setup_ms": float(np.mean([p["mean_setup_ms"] for p in parts])),
                "peak_running": max(p["peak_running"] for p in parts),
                "peak_budgeted_bytes": max(p["peak_bytes"] for p in parts), "completed": agg["completed"],
                "failed": sum(p["failed"] for p in parts), "wall_s": agg["wall_s"],
                "all_done": all(p["all_done"] for p in parts),
                "peak_cohort": max(p["peak_cohort"] for p in parts),
                "cohort_requests": sum(p["cohort_requests"] for p in parts)}

    # warm-up: one request of every kind and size (kernel loading, first-use costs)
    seen, warm = set(), set()
    for k, r in enumerate(reqs):
        key = (r.kind, r.rbc.Nx if r.rbc else r.N)
        if k in mine and key not in seen:
            seen.add(key)
            warm.add(k)
    replay(8, False, subset=warm)
    # continuous batching: up to 16 requests in flight, chunks of 10 steps;
    # plain GPU form: one request at a time, chunks of 50 steps
    served = replay(16, True)
    plain = replay(1, True, chunk=50)
    # saturated capacity: the host-side plan setup and the shared device make
    # single replays vary by up to 2x, so each form is replayed three times
    # (alternating) and the median run by solves/s is reported; one more run
    # stacks same-shape requests with similar step counts into cohorts (up to
    # 16 members per stacked plan)
    sat_runs, plain_runs = [], []
    for _ in range(3):
        sat_runs.append(replay(16, False))
        plain_runs.append(replay(1, False, chunk=50))
    sat_cohort = replay(16, False, cohort=16)

    def median_run(runs):
        return sorted(runs, key=lambda r: r["solves_per_s"])[len(runs) // 2]

    sat, sat_plain = median_run(sat_runs), median_run(plain_runs)
    sat = dict(sat, runs_solves_per_s=[r["solves_per_s"] for r in sat_runs])
    sat_plain = dict(sat_plain, runs_solves_per_s=[r["solves_per_s"] for r in plain_runs])
    kinds = {"rbc": sum(r.kind == "rbc" for r in reqs), "turb": sum(r.kind == "turb" for r in reqs)}
    return {
        "metric": "serving solves/s and time to solution (Poisson 20/s replay)",
        "value": served["solves_per_s"],
        "unit": "requests/s",
        "requests": len(reqs),
        "mix": kinds,
        "n_gpus": world,
        "sharding": "requests assigned to ranks by cost, each rank replays its share at the original arrival "
                    "times, no collective" if world > 1 else "one GPU",
        "hbm_budget_bytes": budget,
        "replay": served,
        "plain_gpu_replay": plain,
        "saturated": sat,
        "plain_gpu_saturated": sat_plain,
        "saturated_speedup_vs_plain_gpu": sat["solves_per_s"] / max(sat_plain["solves_per_s"], 1e-30),
        "saturated_with_cohorts": {k: sat_cohort[k] for k in ("solves_per_s", "p50_ms", "p99_ms", "mean_setup_ms",
                                                              "peak_running", "peak_cohort", "cohort_requests")},
        "dtype": {"rbc": "f64", "turbulence": "f32"},
        "data": "synthetic: seeded arrivals (seed 11), sizes and parameters; RBC noise seed 5000+k, "
                "turbulence k^-3 spectrum seed 7000+k",
    }


_FP64_PEAK = None


def fp64_peak_tflops():
    global _FP64_PEAK
    if _FP64_PEAK is None:
        import torch

        n = 8192
        a = torch.randn(n, n, dtype=torch.float64, device="cuda")
        b = torch.randn(n, n, dtype=torch.float64, device="cuda")
        for _ in range(2):
            torch.matmul(a, b)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = 1e30
        for _ in range(3):
            e0.record()
            torch.matmul(a, b)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        _FP64_PEAK = 2.0 * n ** 3 / (best / 1e3) / 1e12
        del a, b
    return _FP64_PEAK


def main():
    args = parse_args()
    # The CPU reference leg runs on rank 0 alone and needs no collectives: the
    # other ranks leave at once instead of waiting in a barrier for the
    # minutes of host work on rank 0.
    dist = Dist(collectives=args.impl != "reference")
    if args.gpus is None:
        args.gpus = dist.world
    sys.path.insert(0, os.path.join(ROOT, "tarang.jl_b200"))
    from __graft_entry__ import load_package

    if args.impl == "ours":
        load_package()
    import importlib

    spec = importlib.util.spec_from_file_location("tb_workloads", os.path.join(ROOT, "tarang.jl_b200", "workloads.py"))
    W = importlib.util.module_from_spec(spec)
    sys.modules["tb_workloads"] = W
    spec.loader.exec_module(W)
    cfg = W.C2 if args.config == "c2" else W.C1
    scheme = args.scheme if args.config == "c2" else "RK222"
    try:
        if args.impl == "reference":
            run_reference(args, cfg, scheme, dist)
        elif args.workload == "ensemble":
            res = run_ensemble(args, dist.local, dist)
            if dist.rank == 0:
                print(json.dumps(res), flush=True)
        elif args.workload == "serving":
            res = run_serving(args, dist.local, dist)
            if dist.rank == 0:
                print(json.dumps(res), flush=True)
        elif args.workload == "rbc3d":
            if dist.rank == 0:
                print(json.dumps(run_rbc3d(args, dist.local)), flush=True)
        elif args.workload == "turb":
            if dist.rank == 0:
                print(json.dumps(run_turb(args, dist.local)), flush=True)
        else:
            run_ours(args, cfg, scheme, dist)
    finally:
        dist.close()


if __name__ == "__main__":
    main()
