#!/usr/bin/env python
"""Throughput of the reacting-RANS residual/update step on B200.

Workload (one GPU): the 3-D supersonic H2 / vitiated-air mixing layer,
384 x 192 x 64 = 4.72 M cells, 9 species / 19 reactions, k-omega SST,
DPLUR with 4 sweeps, point-implicit (EPI) chemistry.  Synthetic case data
(grid and tanh-blended initial field generated by openstc_b200.cases).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--mode surrogate|mixed|fp64]

--mode surrogate (default, the headline): FP32-bulk / FP64-critical kernels
with the chemistry surrogate; the network is trained on the GPU (samples
from the flow field after a few steps, labels from the FP64 EPI step) before
the timed steps.  The plain FP64 path runs the same number of steps from the
same initial field, and the line reports the relative L2 difference of T,
Y_OH and p.  --mode mixed: the same kernels without the surrogate; --mode
fp64: the reference's arithmetic.  --workload batched: the 12-block
multi-block grid; --workload ramp: the 2-D laminar ramp (256 x 128, FP64,
5000 steps); --long-steps N: the surrogate path beside the FP64 path for N
steps.

`e2e` is the same metric through the C ABI with host buffers: --e2e-steps
steps of the host-driven loop (ostc_driver_step_io), each step's bv and sv
uploaded from pinned host memory before it and downloaded after it; one
step's download and the next step's upload overlap chunk by chunk.

Prints one JSON line (rank 0).  For N > 1 (torchrun) every rank runs an
independent replica of the workload (the path runs on one GPU; there is no
exchange between ranks) and value = all cells x steps / max-over-ranks time.
`--impl reference` times the reference program itself on the same case:
oracle/_ref/openstc_ref, Liangerty/OpenSTC built from its own sources by
oracle/ref/Makefile (its only implementation of this path is its CUDA build;
it has no CPU path), run for 2K steps; the time per step is the reference's
own step timer over steps K+1..2K, so start-up, file I/O and warm-up stay
outside.  Without that binary the arm times the CPU oracle
(oracle/libostc_oracle.so, OpenMP over all host cores) on a bounded sample of
the workload.
"""
from __future__ import annotations

import argparse
import json
import re
import os
import shutil
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))
sys.path.insert(0, str(ROOT / "tests"))

METRIC = "reacting-RANS Mcell*steps/s: FP32+surrogate vs plain FP64 at 1e-3 rel. L2"
UNIT = "Mcell*steps/s"

# DRAM bytes per cell of one launch, from ncu (dram__bytes_read.sum +
# dram__bytes_write.sum) on the 128x64x32 case, scaled by cells: the FP64
# kernels, and the FP32-bulk kernels with every cell's chemistry
# point-implicit (the surrogate's quiet cells are taken off below).  The sweep's
# is the mean of a step's four.
KERNEL_TRAFFIC = {
    "fp64": {"flux": 699.0, "dplur_sweep": 1415.0, "source": 925.0, "dq0": 1415.0, "sweep_terms": 241.0},
    "mixed": {"flux_x": 408.0, "flux_y": 476.0, "flux_z": 444.0, "dplur_sweep": 934.0, "source": 730.0, "dq0": 1123.0,
              "sweep_terms": 197.0},
}
# what a cell that is quiet under the surrogate saves an FP32-bulk sweep: the
# factors and pivots, from captures with none and 14.1 % of the cells quiet
TRAFFIC_EPI = {"dplur_sweep": 631.0}

# Algorithmic bytes per cell of each kernel (9 species, SST, EPI, DPLUR): every
# array a kernel needs, counted once per launch.

# The FP32-bulk path's kernels that read other operands than the FP64 path's,
# counted the same way; a quad is four FP32 components of a cell.  A sweep reads
# of its neighbours' state 8 quads (metric 3, rho u v w, Y 2 1/4, the turbulence
# scalars), the quad of spectral radii and total enthalpy, the pressure term
# and the increments in FP32 (16), of its own dq0 (16 FP32), dt and the SST
# Jacobian (1 + 2 FP64) and the quiet flag; it writes FP32 increments and their
# pressure term from nine weights and a quad with gamma, the last of four
# sweeps the FP64 dq instead.  dq0 reads dq (16), dt, the radii and the SST
# Jacobian in FP64 and writes dq0 in FP32; sweep_terms reads dq0, a quad, T,
# gamma, Y and the radii and writes the nine weights, the quad of radii and the
# pressure term.  A flux pass reads the 11 quads of its operands and adds to dq.
# EPI_BYTES: what each cell whose chemistry stays point-implicit adds (the
# surrogate's quiet cells skip it): the sweep reads the EPI factors of the 8 x 8
# block (64 FP64) and the pivots (8 B); dq0 reads the EPI Jacobian block and
# writes the factors and pivots.
KERNEL_BYTES_MIXED = {
    "dplur_sweep": (16 * 9 + 4 + 4 * 16) + (4 * 16 + 8 * (1 + 2) + 1) + (3 * (4 * 17 + 4 * 9 + 16) + 8 * 16) / 4,
    "dq0": 8 * (16 + 1 + 3 + 2) + 4 * 16 + 1,
    "sweep_terms": (4 * 16 + 16 + 8 * (2 + 9 + 3)) + (4 * 9 + 16 + 4),
    "flux_x": 16 * 11 + 8 * (32 + 4 + 1),
    "flux_y": 16 * 11 + 8 * 32,
    "flux_z": 16 * 11 + 8 * 32,
}
EPI_BYTES = {"dplur_sweep": 8 * 64 + 8, "dq0": 2 * 8 * 64 + 8}

KERNEL_BYTES = {
    "source": 8 * (29 + 101),
    "flux": 8 * (59 + 21),
    # dq 16, the Jacobian 81, dt, the radii 3 and the SST Jacobian 2; dq0, the
    # factors and pivots
    "dq0": 8 * (103 + 97) + 9,
    # dq0 16, u v w |V| T gamma, Y 9; h_k 9 and the three terms
    "sweep_terms": 8 * (31 + 12),
    # metric 9, u v w, Y and the turbulence scalars 11, the three terms, radii 3,
    # increments and dq0 32, dt, factors 81, SST Jacobian 2; three sweeps of four
    # also |V|, T, gamma and h_k for the two pressure terms they write
    "dplur_sweep": 8 * (145 + 16 + (12 + 2) * 3 / 4) + 9,
    "update": 8 * (40 + 34),
    "properties": 8 * (11 + 15),
    "limit_flow": 4,
}


# Device memory of a driver per cell of 384x192x64, ghosts included
FP64_STATE, MIXED_STATE = 1857, 2185

# Tensor-core FLOPs of one cell through the network as the fused kernel runs
# it (K of the first layer padded to 16, N of the output layer to 16):
# 2 (16*256 + 3*256*256 + 256*16).
SURROGATE_FLOP_PER_CELL = 2 * (16 * 256 + 3 * 256 * 256 + 256 * 16)


def workload(size: tuple[int, int, int]) -> str:
    """The workload's name, the same on both arms."""
    cells = size[0] * size[1] * size[2]
    return (f"mixing layer {size[0]}x{size[1]}x{size[2]} ({cells} cells), 9 species/19 reactions, k-omega SST, "
            "DPLUR 4 sweeps, point-implicit chemistry")


def host_cpu() -> dict:
    """The host's CPU model and logical core count (nproc)."""
    model = "unknown"
    try:
        for line in Path("/proc/cpuinfo").read_text().splitlines():
            if line.startswith("model name"):
                model = line.split(":", 1)[1].strip()
                break
    except OSError:
        pass
    return {"cpu_model": model, "nproc": os.cpu_count() or 1}


def parse_size(s: str) -> tuple[int, int, int]:
    a = [int(v) for v in s.lower().split("x")]
    return a[0], a[1], a[2]


def ensure_case(size: tuple[int, int, int], steps_hint: int, base: Path | None = None) -> Path:
    from openstc_b200 import cases

    mx, my, mz = size
    case = (base or ROOT / "cases") / f"bench_ml_{mx}x{my}x{mz}"
    marker = case / ".ready"
    if not marker.exists():
        cases.mixing_layer_case(case, mx=mx, my=my, mz=mz, total_step=10 ** 6, output_screen=1000)
        marker.write_text("ok")
    return case


def shared_case(size: tuple[int, int, int], steps_hint: int, rank: int, world: int, dist,
                base: Path | None = None) -> Path:
    """The case directory every rank reads: rank 0 writes it, the others wait
    at a barrier and then find it (all ranks reach the barrier)."""
    if rank == 0:
        ensure_case(size, steps_hint, base)
    if world > 1:
        dist.barrier()
    return ensure_case(size, steps_hint, base)


def max_over_ranks(ms: float, dist, world: int, device) -> float:
    """The slowest rank's time (ms), the same on every rank; every rank takes
    part in the one collective."""
    import torch

    t = torch.tensor([ms], dtype=torch.float64, device=device)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_rate(cells: int, world: int, steps: int, ms: float) -> float:
    """Mcell*steps/s of the whole job: every rank steps its own replica of
    `cells` cells `steps` times in the (max-over-ranks) time ms."""
    return world * cells * steps / (ms / 1e3) / 1e6


class ClockSampler:
    """nvidia-smi clock / throttle samples while the timed region runs."""

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.rows: list[list[str]] = []
        self._p = None

    def __enter__(self):
        q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        try:
            self._p = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                        "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self._t = threading.Thread(target=self._read, daemon=True)
            self._t.start()
        except FileNotFoundError:
            self._p = None
        return self

    def _read(self):
        for line in self._p.stdout:
            self.rows.append([v.strip() for v in line.split(",")])

    def __exit__(self, *a):
        if self._p:
            self._p.terminate()
            self._p.wait()

    def summary(self) -> dict:
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[0]) for r in self.rows if r[0].replace(".", "").isdigit()]
        mx = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self.rows for i in range(4) if len(r) > 3 + i and r[3 + i] == "Active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


def peaks() -> dict:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return {"hbm_gbs": d["hbm_gbs"], "bf16_tflops": d.get("bf16_tflops"),
                "bf16_tflops_sustained": d.get("bf16_tflops_sustained"), "source": "measured"}
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0, "source": "fallback"}


def cpu_sample(threads: int, seconds: float = 15.0) -> dict:
    """The CPU oracle on a bounded sample of the workload: same physics,
    a 48 x 24 x 16 grid, steps until `seconds` have passed."""
    import openstc_b200 as ostc
    from oracle_bridge import OracleSolver

    case = ensure_case((48, 24, 16), 0)
    orc = OracleSolver(ostc.Driver(case), threads=threads)
    orc.initialize()
    cells = 48 * 24 * 16
    t0 = time.perf_counter()
    n = 0
    while True:
        n += 1
        orc.step(n + 1)  # step numbers past 1 and off the residual cadence
        dt = time.perf_counter() - t0
        if dt > seconds:
            break
    return {"value": cells * n / dt / 1e6, "unit": UNIT, "cores": threads,
            "sample": f"48x24x16 cells of the same case, {n} steps in {dt:.1f} s (FP64 oracle)"}


REF_BIN = ROOT / "oracle" / "_ref" / "openstc_ref"


def _reference_run(case: Path, steps: int, work: Path, screen: int = 10 ** 7) -> float:
    """Wall seconds of one run of the reference program on a copy of `case`
    stopped after `steps` steps, printing its residual and its own step timer
    every `screen` steps (run.log in the run's directory)."""
    d = work / f"run_{steps}"
    if d.exists():
        shutil.rmtree(d)
    (d / "input_files").mkdir(parents=True)
    for sub in (case / "input_files").iterdir():
        if sub.name == "setup":
            shutil.copytree(sub, d / "input_files" / "setup")
        else:
            (d / "input_files" / sub.name).symlink_to(sub.resolve())
    shutil.copytree(case / "output", d / "output")
    ctl = d / "input_files" / "setup" / "0_global_control.txt"
    lines = []
    for line in ctl.read_text().splitlines():
        key = line.split("=")[0].split()
        if len(key) == 2 and key[0] == "int" and key[1] in ("total_step", "output_screen", "output_file"):
            val = steps if key[1] == "total_step" else (screen if key[1] == "output_screen" else 10 ** 7)
            line = f"int {key[1]} = {val}"
        lines.append(line)
    ctl.write_text("\n".join(lines) + "\n")
    with open(d / "run.log", "w") as log:
        t0 = time.perf_counter()
        subprocess.run([str(REF_BIN)], cwd=d, stdout=log, stderr=subprocess.STDOUT, timeout=3600, check=True)
        return time.perf_counter() - t0


def batched_case(seed: int) -> Path:
    """The batched multi-block workload: the mixing-layer physics on 12
    seeded blocks tiled along x (cases.batched_multiblock_case)."""
    from openstc_b200 import cases

    case = ROOT / "cases" / f"bench_batched_seed{seed}"
    if not (case / ".ready").exists():
        cases.batched_multiblock_case(case, seed=seed, total_step=10 ** 6, output_screen=1000)
        (case / ".ready").write_text("ok")
    return case


def batched_workload(seed: int) -> tuple[str, int]:
    from openstc_b200 import cases

    mxs, my, mz = cases.batched_block_sizes(seed)
    cells = sum(mxs) * my * mz
    return (f"batched multi-block: 12 blocks (seed {seed}) of mx in {min(mxs)}..{max(mxs)} x {my} x {mz} tiled "
            f"along x ({cells} cells), mixing-layer physics, 9 species/19 reactions, k-omega SST, DPLUR 4 sweeps, "
            "point-implicit chemistry"), cells


def batched_arm(args) -> None:
    """The batched multi-block workload on one GPU: the FP64 path with exact
    inner faces (bit-identical to the same grid as one block) and the
    FP32-bulk path after the launch autotuner, each timed over K graph-launched
    steps; value = the FP32-bulk path's rate."""
    import torch

    import openstc_b200 as ostc

    torch.cuda.set_device(0)
    case = batched_case(args.seed)
    name, cells = batched_workload(args.seed)
    W, K = max(args.warmup, 3), args.steps
    out = {}
    for label, kw in (("fp64_exact", dict(precision="fp64", exact_inner=True)), ("mixed", dict(precision="mixed"))):
        drv = ostc.Driver(case, **kw)
        drv.initialize()
        tuning = drv.autotune(reps=2)
        drv.step(W)
        ms, clocks = timed_steps(drv, K, torch, 0, None, 1, "timed_batched_" + label)
        out[label] = {"ms_per_step": ms / K, "value": cells * K / (ms / 1e3) / 1e6, "tuning": tuning,
                      "clocks": clocks, "launches_per_step": drv.launches_per_step(False, False)}
        drv.close()
    line = {"metric": METRIC, "value": out["mixed"]["value"], "unit": UNIT, "n_gpus": 1, "steps": K, "warmup": W,
            "ms_per_step": out["mixed"]["ms_per_step"], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
            "config": {"workload": name, "path": "mixed", "parallelism": "replicas x1"},
            "fp64_exact_inner": out["fp64_exact"], "mixed": out["mixed"], "clocks": out["mixed"]["clocks"]}
    print(json.dumps(line), flush=True)


RAMP_SIZE = (256, 128)
RAMP_METRIC = "laminar ramp Mcell*steps/s, FP64"


def ramp_case_dir() -> Path:
    """The plain-method workload: 2-D laminar air at Mach 3 over a 15 degree
    compression ramp, one 256 x 128 block (cases.ramp_case)."""
    from openstc_b200 import cases

    case = ROOT / "cases" / f"bench_ramp_{RAMP_SIZE[0]}x{RAMP_SIZE[1]}"
    if not (case / ".ready").exists():
        cases.ramp_case(case, mx=RAMP_SIZE[0], my=RAMP_SIZE[1], total_step=10 ** 6, output_screen=1000,
                        output_file=10 ** 7)
        (case / ".ready").write_text("ok")
    return case


def ramp_workload() -> tuple[str, int]:
    cells = RAMP_SIZE[0] * RAMP_SIZE[1]
    return (f"laminar ramp {RAMP_SIZE[0]}x{RAMP_SIZE[1]} ({cells} cells): 2-D air, Mach 3, 2.5 kPa, 220 K over a 15 "
            "degree compression ramp, isothermal 300 K wall, AUSM+/MUSCL-minmod, explicit Euler with local time "
            "step at CFL 0.5, FP64"), cells


def ramp_arm(args) -> None:
    """The plain-method workload on one GPU, the reference's arithmetic (FP64):
    the launch autotuner's choice of flux kernel, then --ramp-steps
    graph-launched steps (the workload's 5000 by default) with the residual
    every 1000 steps, CUDA events around them, after W warm-up steps.  The
    grid (32 k cells) is far smaller than L2: this measures the launch-bound
    step the CUDA graph serves, not HBM."""
    import torch

    import openstc_b200 as ostc

    torch.cuda.set_device(0)
    case = ramp_case_dir()
    name, cells = ramp_workload()
    W, K = max(args.warmup, 3), args.ramp_steps
    drv = ostc.Driver(case, precision="fp64")
    drv.initialize()
    tuning = drv.autotune(reps=20)
    drv.step(W)
    ms, clocks = timed_steps(drv, K, torch, 0, None, 1, "timed_ramp")
    line = {"metric": RAMP_METRIC, "value": cells * K / (ms / 1e3) / 1e6, "unit": UNIT, "n_gpus": 1, "steps": K,
            "warmup": W, "ms_per_step": ms / K, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic",
            "config": {"workload": name, "path": "fp64", "parallelism": "replicas x1",
                       "l2": "inputs smaller than L2 (32 k cells, launch-bound)"},
            "clocks": clocks, "gpu_launches": drv.launches_per_step(False, False) * K, "tuning": tuning}
    drv.close()
    print(json.dumps(line), flush=True)


def long_arm(args) -> None:
    """The full chosen form over a long run: the FP32-bulk path with the
    chemistry surrogate (trained on the flow field after --snapshot-steps
    steps) beside the plain FP64 path on the same GPU, both from the same
    initial field, stepped in lockstep for --long-steps steps.  Records both
    residual histories (every 10 steps), the relative L2 of T, Y_OH and p
    between the paths at 500, 1000, 2000, ... steps, the fallback fraction and
    each path's Mcell*steps/s (CUDA events over its own steps)."""
    import torch

    import openstc_b200 as ostc
    from openstc_b200 import cases

    torch.cuda.set_device(0)
    size = parse_size(args.size)
    case = ROOT / "cases" / f"long_ml_{size[0]}x{size[1]}x{size[2]}"
    if not (case / ".ready").exists():
        cases.mixing_layer_case(case, mx=size[0], my=size[1], mz=size[2], total_step=10 ** 6, output_screen=10)
        (case / ".ready").write_text("ok")
    S = max(args.snapshot_steps, 1)
    ref = ostc.Driver(case, precision="fp64")
    ref.initialize()
    drv = ostc.Driver(case, precision="mixed")
    drv.initialize()
    cells = ref.info().n_grid_total
    hist = {"fp64": [], "surrogate": []}
    ms = {"fp64": 0.0, "surrogate": 0.0}

    def advance(d, name, n):
        stream = torch.cuda.ExternalStream(d.stream())
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record(stream)
        err = d.step(n)
        b.record(stream)
        torch.cuda.synchronize()
        ms[name] += a.elapsed_time(b)
        return err

    for name, d in (("fp64", ref), ("surrogate", drv)):
        hist[name].append([1, advance(d, name, 1)])
        advance(d, name, S - 1) if S > 1 else None
    sur = ostc.Surrogate(drv, seed=1234)
    t0 = time.perf_counter()
    sur.generate(args.samples, seed=77, field=drv, field_fraction=args.field_fraction)
    sur.train(args.train_steps, batch=65536, lr=2e-3, n_train=args.samples - (1 << 18))
    held = sur.evaluate(args.samples - (1 << 18), 1 << 18)
    train_s = time.perf_counter() - t0
    drv.set_surrogate(sur)
    checkpoints = {}
    step = S
    while step < args.long_steps:
        n = min(10 - step % 10, args.long_steps - step)
        for name, d in (("fp64", ref), ("surrogate", drv)):
            e = advance(d, name, n)
            if (step + n) % 10 == 0:
                hist[name].append([step + n, e])
        step += n
        if step in (500, 1000, 1500, 2000, 3000, 4000, 5000) or step == args.long_steps:
            checkpoints[step] = rel_l2(interior_fields(drv), interior_fields(ref))
    a, f = drv.chemistry_stats()
    line = {"metric": METRIC, "unit": UNIT, "n_gpus": 1, "steps": args.long_steps, "data": "synthetic",
            "config": {"workload": workload(size), "path": "surrogate beside fp64", "lockstep": True},
            "value": cells * (args.long_steps - S) / (ms["surrogate"] / 1e3) / 1e6 if ms["surrogate"] else None,
            "fp64_value": cells * args.long_steps / (ms["fp64"] / 1e3) / 1e6,
            "accuracy_vs_fp64": {str(k): v for k, v in checkpoints.items()},
            "chemistry": {"accepted": a, "fallback": f, "fallback_fraction": f / max(1, a + f)},
            "surrogate_training": {"samples": args.samples, "steps": args.train_steps, "seconds": train_s,
                                   "held_out": {k: held[k] for k in ("median_rel_all", "p90_rel_all", "gate_pass")},
                                   "gate": sur.gate()},
            "residual_history": hist}
    print(json.dumps(line), flush=True)
    drv.set_surrogate(None)
    drv.close()
    ref.close()
    sur.close()


def reference_arm(args) -> None:
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    gpu = shutil.which("nvidia-smi") is not None and subprocess.run(
        ["nvidia-smi", "-L"], capture_output=True).returncode == 0
    if REF_BIN.exists() and gpu:
        metric = METRIC
        if args.workload == "batched":
            case = batched_case(args.seed)
            name, cells = batched_workload(args.seed)
            work = ROOT / "cases" / "reference_arm_batched"
        elif args.workload == "ramp":
            case = ramp_case_dir()
            name, cells = ramp_workload()
            work = ROOT / "cases" / "reference_arm_ramp"
            metric = RAMP_METRIC
        else:
            size = parse_size(args.size)
            case = ensure_case(size, args.steps)
            name, cells = workload(size), size[0] * size[1] * size[2]
            work = ROOT / "cases" / "reference_arm"
        # The reference times itself between residual prints (gxl::Time,
        # MPI_Wtime): with a print every K steps over 2K steps, its last
        # "CPU time for this step" covers steps K+1..2K -- the first K are the
        # warm-up -- with no start-up or file I/O inside.
        K = args.ramp_steps if args.workload == "ramp" else max(args.steps, args.warmup, 1)
        wall = _reference_run(case, 2 * K, work, screen=K)
        found = re.findall(r"CPU time for this step is\s+([0-9.eE+-]+)s", (work / f"run_{2 * K}" / "run.log").read_text())
        if found:
            sec = float(found[-1])
            sample = (f"reference CUDA program (oracle/_ref/openstc_ref) on the GPU, same case; its own timer over "
                      f"steps {K + 1}-{2 * K} of a {2 * K}-step run ({wall:.1f} s wall with start-up)")
            steps = K
        else:
            w = max(args.warmup, 1)
            t_w = _reference_run(case, w, work)
            t_wk = _reference_run(case, w + args.steps, work)
            sec = max(t_wk - t_w, 1e-9)
            steps = args.steps
            sample = (f"reference CUDA program (oracle/_ref/openstc_ref) on the GPU, same case; "
                      f"{w + args.steps}-step run {t_wk:.2f} s minus {w}-step run {t_w:.2f} s")
        value = cells * steps / sec / 1e6
        line = {"impl": "reference", "metric": metric, "value": value, "unit": UNIT, "n_gpus": args.gpus,
                "steps": steps, "warmup": args.warmup, "ms_per_step": 1e3 * sec / steps,
                "higher_is_better": True, "dtype": "f64", "data": "synthetic",
                "config": {"workload": name, "path": "reference CUDA program, FP64",
                           "parallelism": "replicas x1",
                           "l2": "inputs smaller than L2 (32 k cells, launch-bound)" if args.workload == "ramp"
                           else f"inputs larger than L2 (state ~{cells * 1650 / 1e9:.1f} GB)"},
                "cpu_baseline": {"kind": "reference", "cores": 1, "sample": sample, "value": value, "unit": UNIT}
                | host_cpu(),
                "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line), flush=True)
        return
    threads = os.cpu_count() or 1
    base = cpu_sample(threads, seconds=max(5.0, 3.0 * args.steps))
    line = {"impl": "reference", "metric": METRIC, "value": base["value"], "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "higher_is_better": True, "dtype": "f64",
            "data": "synthetic", "config": {"workload": workload(parse_size(args.size)),
                                            "path": "CPU oracle on a bounded sample"},
            "cpu_baseline": {"kind": "port", "cores": threads, "sample": base["sample"], "value": base["value"]}
            | host_cpu(),
            "e2e": {"value": base["value"], "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def interior_fields(drv) -> dict:
    """T, Y_OH, p of every interior cell of block 0 (host copies)."""
    g = drv.info().ngg
    bv = drv.get(0, "bv")[:, g:-g, g:-g, g:-g]
    sv = drv.get(0, "sv")[:, g:-g, g:-g, g:-g]
    return {"T": bv[5].copy(), "Y_OH": sv[4].copy(), "p": bv[4].copy()}


def rel_l2(a: dict, b: dict) -> dict:
    return {k: float(np.linalg.norm(a[k] - b[k]) / np.linalg.norm(b[k])) for k in b}


def timed_steps(drv, steps: int, torch, local: int, dist, world: int, label: str = "timed"):
    """CUDA-event time of `steps` graph-launched steps on the engine stream,
    max over ranks; clock samples taken meanwhile.  The steps sit in an NVTX
    range named `label` (a profiler can restrict itself to them)."""
    stream = torch.cuda.ExternalStream(drv.stream())
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clk:
        torch.cuda.nvtx.range_push(label)
        start.record(stream)
        drv.step(steps)
        stop.record(stream)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_pop()
    return max_over_ranks(start.elapsed_time(stop), dist, world, "cuda"), clk.summary()


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--mode", default="surrogate", choices=["surrogate", "mixed", "fp64"],
                    help="surrogate: FP32-bulk/FP64-critical kernels with the chemistry surrogate (the headline); "
                         "mixed: the same without the surrogate; fp64: the reference's arithmetic")
    ap.add_argument("--size", default="384x192x64")
    ap.add_argument("--workload", default="mixing_layer", choices=["mixing_layer", "batched", "ramp"],
                    help="mixing_layer: one block of --size (the headline); batched: 12 seeded blocks tiled along x "
                         "(--seed), FP64 with exact inner faces and FP32-bulk after the launch autotuner; ramp: the "
                         "2-D laminar ramp, 256x128, FP64, --ramp-steps steps")
    ap.add_argument("--ramp-steps", type=int, default=5000)
    ap.add_argument("--seed", type=int, default=0)
    ap.add_argument("--long-steps", type=int, default=0,
                    help="> 0: the long run of the surrogate path beside the FP64 path (long_arm) on --size")
    ap.add_argument("--field-fraction", type=float, default=0.95)
    ap.add_argument("--snapshot-steps", type=int, default=5,
                    help="steps run before training the surrogate on the resulting flow field")
    ap.add_argument("--train-steps", type=int, default=8000)
    ap.add_argument("--samples", type=int, default=1 << 24)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--e2e-steps", type=int, default=8)
    args = ap.parse_args()
    if args.impl == "reference":
        reference_arm(args)
        return
    if args.workload == "batched":
        batched_arm(args)
        return
    if args.workload == "ramp":
        ramp_arm(args)
        return
    if args.long_steps > 0:
        long_arm(args)
        return
    import torch
    import torch.distributed as dist

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        from datetime import timedelta

        dist.init_process_group("nccl", timeout=timedelta(seconds=600), device_id=torch.device("cuda", local))
    size = parse_size(args.size)
    case = shared_case(size, args.steps, rank, world, dist)

    import openstc_b200 as ostc

    W, K = max(args.warmup, 3), args.steps
    S = max(args.snapshot_steps, 1) if args.mode == "surrogate" else 0
    total = S + W + K
    precision = "fp64" if args.mode == "fp64" else "mixed"

    # the plain FP64 path over the same steps: the accuracy reference
    ref = ostc.Driver(case, device=local)
    ref.initialize()
    ref.step(S + W)
    ms_fp64, _ = timed_steps(ref, K, torch, local, dist, world, "timed_fp64_reference")
    ref_fields = interior_fields(ref)
    cells = ref.info().n_grid_total
    ref.close()

    drv = ostc.Driver(case, device=local, precision=precision)
    drv.initialize()
    sur = None
    train = None
    if args.mode == "surrogate":
        drv.step(S)
        sur = ostc.Surrogate(drv, seed=1234 + rank)
        t0 = time.perf_counter()
        sur.generate(args.samples, seed=77 + rank, field=drv, field_fraction=args.field_fraction)
        losses = sur.train(args.train_steps, batch=65536, lr=2e-3, n_train=args.samples - (1 << 18))
        held = sur.evaluate(args.samples - (1 << 18), 1 << 18)
        train = {"samples": args.samples, "steps": args.train_steps, "batch": 65536, "seconds": time.perf_counter() - t0,
                 "loss_first": float(losses[0]), "loss_last": float(losses[-1]),
                 "held_out": {k: held[k] for k in ("mean_rel", "max_rel", "rel_count", "max_defect",
                                                    "median_rel_all", "p90_rel_all", "gate_pass", "count")},
                 "gate": sur.gate()}
        drv.set_surrogate(sur)
    drv.step(W)
    ms_max, clocks = timed_steps(drv, K, torch, local, dist, world, "timed_" + args.mode)
    value = whole_job_rate(cells, world, K, ms_max)
    launches = drv.launches_per_step(False, False) * K
    acc = rel_l2(interior_fields(drv), ref_fields) if args.mode != "fp64" else {"T": 0.0, "Y_OH": 0.0, "p": 0.0}
    chem = None
    if sur is not None:
        a, f = drv.chemistry_stats()
        ev = drv.surrogate_evaluations()
        chem = {"accepted": a, "fallback": f, "fallback_fraction": f / max(1, a + f),
                "evaluated_fraction": ev / max(1, a + f)}

    # per-kernel device times of one eager step (roofline of the top kernel)
    prof = drv.profile_step()
    top = max(prof, key=lambda r: r[2])
    pk = peaks()
    kernel_bytes = KERNEL_BYTES | (KERNEL_BYTES_MIXED if args.mode != "fp64" else {})
    if args.mode != "fp64":
        # the EPI block of the cells whose chemistry stayed point-implicit
        quiet = chem["accepted"] / max(1, chem["accepted"] + chem["fallback"]) if chem else 0.0
        kernel_bytes = kernel_bytes | {k: kernel_bytes[k] + v * (1.0 - quiet) for k, v in EPI_BYTES.items()}
    top_bytes = kernel_bytes.get(top[0], 0) * cells * top[1]
    achieved = top_bytes / (top[2] / 1e3) / 1e9 if top[2] > 0 else 0.0

    # end to end through the C ABI with host buffers: the host-driven loop
    # (ostc_driver_step_io) uploads each step's state from pinned host
    # memory, steps, and reads the state back into the same buffers; the next
    # step's upload of a chunk follows the download of that chunk
    bv_shape = drv.field_shape(0, "bv")
    sv_shape = drv.field_shape(0, "sv")
    bv_h = torch.empty(int(np.prod(bv_shape)), dtype=torch.float64, pin_memory=True).numpy()
    sv_h = torch.empty(int(np.prod(sv_shape)), dtype=torch.float64, pin_memory=True).numpy()
    drv.get_into(0, "bv", bv_h)
    drv.get_into(0, "sv", sv_h)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    drv.step_io(args.e2e_steps, 0, ["bv", "sv"], [bv_h, sv_h])
    torch.cuda.synchronize()
    # the slowest rank's time per step, as for `value`
    e2e_s = max_over_ranks((time.perf_counter() - t0) / args.e2e_steps * 1e3, dist, world, "cuda") / 1e3
    h2d = (bv_h.nbytes + sv_h.nbytes)

    dtype = {"surrogate": "f32+f64+bf16", "mixed": "f32+f64", "fp64": "f64"}[args.mode]
    traffic_table = dict(KERNEL_TRAFFIC["fp64" if args.mode == "fp64" else "mixed"])
    if args.mode != "fp64" and chem:
        q = chem["accepted"] / max(1, chem["accepted"] + chem["fallback"])
        for k, v in TRAFFIC_EPI.items():
            traffic_table[k] -= v * q
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": K, "warmup": W,
        "ms_per_step": ms_max / K, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": dtype, "data": "synthetic",
        "config": {"workload": workload(size), "path": args.mode, "parallelism": f"replicas x{world}",
                   "l2": f"inputs larger than L2 (state ~{cells * (FP64_STATE if args.mode == 'fp64' else MIXED_STATE) / 1e9:.1f} GB)",
                   "compared_after_steps": total},
        "accuracy_vs_fp64": {"rel_l2": acc, "bar": 1e-3, "within": all(v <= 1e-3 for v in acc.values())},
        "fp64_ms_per_step": ms_fp64 / K,
        "clocks": clocks,
        "gpu_launches": launches,
        "kernels_ms_per_step": {n: round(v, 4) for n, _, v in prof},
        "roofline": {"bound": "hbm", "kernel": top[0], "achieved": achieved, "peak": pk["hbm_gbs"], "unit": "GB/s",
                     "frac": achieved / pk["hbm_gbs"],
                     "traffic": traffic_table[top[0]] * cells if top[0] in traffic_table else None,
                     "peak_source": pk["source"], "bytes_per_cell": round(kernel_bytes.get(top[0], 0), 1)},
        "e2e": {"value": world * cells / e2e_s / 1e6, "unit": UNIT, "h2d_bytes_per_step": h2d,
                "d2h_bytes_per_step": h2d},
    }
    if chem is not None:
        line["chemistry"] = chem
        sur_ms = sum(v for n, _, v in prof if n == "surrogate")
        if sur_ms > 0:
            # the fused inference: tensor-core bound, timed inside a long step
            # the cells the network evaluates in a step (quiet ones and a
            # rotating share of the rest)
            flops = SURROGATE_FLOP_PER_CELL * cells * chem["evaluated_fraction"]
            tf = flops / (sur_ms / 1e3) / 1e12
            peak_tf = pk.get("bf16_tflops_sustained") or pk.get("bf16_tflops")
            line["roofline_surrogate"] = {"bound": "tensor", "kernel": "surrogate", "achieved": tf, "peak": peak_tf,
                                          "unit": "TFLOP/s", "frac": tf / peak_tf if peak_tf else None,
                                          "flop_per_cell": SURROGATE_FLOP_PER_CELL, "peak_source": pk["source"]}
    if train is not None:
        line["surrogate_training"] = train
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_sample(1, seconds=15.0) | {"kind": "port"} | host_cpu()
    if rank == 0:
        print(json.dumps(line), flush=True)
    drv.close()
    if sur is not None:
        sur.close()
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
