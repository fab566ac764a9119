"""Benchmark of the GB300 MONKI transport hot path.

Default workload: the 3-D box cloud (polarized I/Q/U): 30 x 20 periodic 1 km columns, 34
layers plus vacuum, Rayleigh 0.70 + O3 0.30 + aerosol 0.20 (g 0.70, SSA 0.92), a 10 x 6
column cloud block at 1-3 km of optical depth 20 (g 0.85, SSA 0.9999), SZA 60, views
(VZA, RAA) = (0,0), (30,90), (60,180), albedo 0.05, FP32 transport with FP64 per-round
tallies, 50,000 photons per column per round. One step = one statistical round
(30,000,000 photon histories) through the transport kernels and the FP64 flush.
``--workload layered`` runs the layered-cloud scene instead (cloud slab at 2-3 km,
optical depth 10, SZA 30, layer AMF paths, 20,000 photons per column).

Printed JSON (one line, rank 0):
  value      scatters/s of the analog kernels with the scene resident on the device, from
             CUDA events on the session stream (L2 flushed before the timed group);
  time_to_target  wall seconds of ``simulate`` through the public API until SE/|I| < 1 %
             in every pixel and view (standard error of the round means, defined from the
             31st round on), analog and importance-guided, from the same rounds' tallies;
  e2e        scatters/s of that analog ``simulate`` run (host tables in, every round's
             FP64 tallies out, statistics on the host);
  roofline   the peel kernel's algorithmic bytes per launch (event state, cell records of
             the detector rays, 128-bit tally atomics) over its event-timed duration,
             against the measured HBM copy bandwidth;
  cpu_baseline  the FP64 CPU restatement of the reference transport (oracle) on a bounded
             sample of the same round, on every host core.

``--impl reference`` times that CPU restatement alone (the reference's Fortran transport
cannot be compiled here), with the same metric and configuration.
"""

from __future__ import annotations

import argparse
import ctypes
import json
import os
import re
import statistics
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))
sys.path.insert(0, str(ROOT / "monki-gpu_gb300"))

METRIC = "time to SE/|I|<1% per scene, plain vs importance-guided MC on 1 GB300; scatters/s"
UNIT = "scatters/s"
WORKLOADS = {
    "box": ("box_cloud", 50_000, "box-cloud 30x20x35, I/Q/U, SZA 60, 50000 photons/column/round"),
    "layered": ("layered_cloud", 20_000, "layered-cloud 30x20x35, I/Q/U + layer AMF, 20000 photons/column/round"),
}
TARGET = 0.01  # SE/|I| in every pixel and view
# The time-to-target runs use rounds of 2,000 photons per column, checked every round from
# round 32: at this round size the rule decides (the analog run needs about 40 rounds),
# where at the workload's 50,000 every method met the target at its first check. Three
# seeds per method; medians are reported.
# 1,000 photons per column per round: every method needs more than the rule's 32-round
# minimum (at 2,000 the guided methods stop at the minimum, which caps their speed-up).
TARGET_PPC = 1000
TARGET_SEEDS = (23274, 23275, 23276)
TARGET_CAP = 1024  # round cap of a time-to-target run
# epsilon, roulette weight, cap, split: Russian roulette below weight 0.25, splitting above 0.5
# (the fastest constant weight window to the target of a sweep of roulette 0.2-1 and split
# 1.5-3 on this scene).
GUIDED = (0.0, 0.25, 0.0, 2.0)
E2E_ROUNDS = 32  # rounds of the end-to-end run at the workload's own round size
STATE_BYTES = 64  # one event's photon state records read by the peel kernel
CELL_BYTES = 16  # one cell record (beta + cumulative species fractions)
TALLY_BYTES = 32  # one 128-bit tally atomic: 16 B read + 16 B written in L2
TRANSIT_EVENT_BYTES = 109  # per event: state read (52 B) and written (52 B), queue entry and kind (5 B)
SCATTER_EVENT_BYTES = 116  # per event: queue entry (4 B), state read (64 B) and written (48 B)
# Fused step (scenes without layer paths): per event its list entry (4 B), its state read once
# (64 B) and written once after the walk (52 B), its new queue entry and kind (5 B) — the
# algorithmic minimum; the measured DRAM traffic adds what misses L2 (a record block read by
# the peel-off is read again by the next step) and walks paused by the step budget.
STEP_EVENT_BYTES = 125


def peaks():
    path = ROOT / "MEASURED_PEAKS.json"

    if path.is_file():
        data = json.loads(path.read_text())
        return float(data["hbm_gbs"]), "measured"

    return 6800.0, "fallback"


def recorded_traffic(workload, kernel, per_launch=None):
    """Per-launch DRAM bytes (read + write) of one wavefront kernel from the committed ncu
    summary of the workload, or None. The captures ran fewer photons per column than the
    bench's launches; when the summary gives the algorithmic bytes of the captured launch, its
    traffic is scaled to this launch by the algorithmic bytes (the units processed): the
    traffic grows with the events a launch handles."""

    name = {"box": "box_cloud", "layered": "layered_cloud"}[workload]
    path = ROOT / "profiles" / f"transport_kernel_{name}.md"

    if not path.is_file():
        return None

    text = path.read_text()
    match = re.search(rf"traffic_{kernel}_bytes_per_launch:\s*([0-9.eE+]+)", text)
    if match is None and kernel == "peel":
        match = re.search(r"traffic_bytes_per_launch:\s*([0-9.eE+]+)", text)
    if match is None:
        return None
    traffic = float(match.group(1))
    captured = re.search(rf"algorithmic_{kernel}_bytes_per_captured_launch:\s*([0-9.eE+]+)", text)
    if captured is not None and per_launch:
        traffic *= per_launch / float(captured.group(1))
    return traffic


class Clocks:
    """nvidia-smi samples of SM clock and throttle reasons during the timed region."""

    QUERY = (
        "index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
        "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
        "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap"
    )

    def __init__(self, device: int):
        self.device = device
        self.process = None
        self.path = Path(os.environ.get("TMPDIR", "/tmp")) / f"monki_clocks_{os.getpid()}.csv"

    def __enter__(self):
        try:
            self.process = subprocess.Popen(
                ["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"),
                stderr=subprocess.DEVNULL,
            )
        except (FileNotFoundError, OSError):
            self.process = None

        return self

    def __exit__(self, *args):
        if self.process is not None:
            self.process.terminate()
            try:
                self.process.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.process.kill()

    def summary(self):
        if self.process is None or not self.path.is_file():
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}

        rows = []

        for line in self.path.read_text().splitlines():
            parts = [p.strip() for p in line.split(",")]

            if len(parts) >= 9:
                rows.append(parts)

        self.path.unlink(missing_ok=True)

        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}

        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        top = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        reasons = sorted({name for r in rows for name, flag in zip(names, r[5:9]) if flag.lower() == "active"})
        loaded = sorted(sm)[len(sm) // 2 :] or sm
        return {
            "sm_mhz": statistics.median(loaded) if loaded else None,
            "sm_max_mhz": max(top) if top else None,
            "reasons": reasons,
            "samples": len(rows),
        }


def distributed():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


ROUNDS_PER_RANK = 100000  # rank r runs statistical rounds from r * 100000 + 1: disjoint streams


def first_round(rank: int, round_in_rank: int) -> int:
    """The global round index of a rank's round: ranks never share a Philox stream."""

    return rank * ROUNDS_PER_RANK + round_in_rank


def combine_ranks(seconds: float, scatters: float, device):
    """Whole-job timing and work over the ranks of the process group: the slowest rank's
    device seconds and the summed scatters (the only exchange; no data-path collective)."""

    import torch
    import torch.distributed as dist

    t = torch.tensor([seconds], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    s = torch.tensor([float(scatters)], device=device, dtype=torch.float64)
    dist.all_reduce(s)
    return float(t.item()), float(s.item())


def cpu_baseline(scene, target_seconds: float = 10.0):
    """Scatters/s of the FP64 CPU restatement on a bounded sample of one round."""

    from oracle import oracle

    nmat, nx, ny, nz, angles = scene.shape
    per_round = scene.photons_per_column * nx * ny
    threads = os.cpu_count() or 1
    calibration = max(threads * 64, 4096)
    start = time.perf_counter()
    _, counters = oracle.run(scene.tables, [calibration, 0, 1, 0, 100000, 0, per_round, 1], threads)
    rate = calibration / max(time.perf_counter() - start, 1e-6)
    sample = int(min(per_round - calibration, max(calibration, rate * target_seconds)))
    start = time.perf_counter()
    _, counters = oracle.run(scene.tables, [sample, calibration, 1, 0, 100000, 0, per_round, 1], threads)
    elapsed = time.perf_counter() - start
    return {
        "value": counters["scatters"] / elapsed,
        "unit": UNIT,
        "cores": threads,
        "kind": "port",
        "sample": f"{sample} of the {per_round} photon histories of one round ({elapsed:.1f} s, "
        f"{counters['scatters']} scatters), FP64 C++ restatement of mc.f90 with OpenMP",
    }


def build_scene(workload, photons_per_column, rounds):
    import monki.scenes as scenes

    builder, _, _ = WORKLOADS[workload]
    return getattr(scenes, builder)(photons_per_column, rounds)


def reference_arm(args):
    world, rank, _ = distributed()

    if rank != 0:
        return 0

    from oracle import oracle

    _, default_ppc, workload = WORKLOADS[args.workload]
    ppc = args.photons_per_column or default_ppc
    scene = build_scene(args.workload, ppc, 1)
    nmat, nx, ny, nz, angles = scene.shape
    per_round = ppc * nx * ny
    threads = os.cpu_count() or 1
    sample = max(threads * 256, 20_000)
    scatters = 0
    elapsed = 0.0

    for step in range(args.warmup + args.steps):
        first = (step * sample) % max(per_round - sample, 1)
        start = time.perf_counter()
        _, counters = oracle.run(scene.tables, [sample, first, 1, 0, 100000, 0, per_round, 1], threads)
        dt = time.perf_counter() - start

        if step >= args.warmup:
            scatters += counters["scatters"]
            elapsed += dt

    value = scatters / elapsed
    line = {
        "impl": "reference",
        "metric": METRIC,
        "value": value,
        "unit": UNIT,
        "n_gpus": args.gpus,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": elapsed / args.steps * 1e3,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f64",
        "data": "synthetic",
        "config": {"workload": workload, "step": f"{sample} photon histories of one round on the host cores"},
        "cpu_baseline": {
            "value": value,
            "unit": UNIT,
            "cores": threads,
            "kind": "port",
            "sample": f"{sample} photon histories per step; the reference's Fortran transport needs gfortran, "
            "which is absent, so its FP64 C++ restatement (oracle/) runs instead",
        },
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


def time_to_target(workload, ppc, device, seed, guided, scale=None):
    """Wall seconds of ``simulate`` (the public API, host tables in, FP64 round statistics on
    the device) until SE/|I| < TARGET in every pixel and view, checked every round from
    round 32; ``guided`` is a Guided or None (analog)."""

    import tempfile

    from monki import RadianceConvergence, simulate
    from monki.execution import CUDA

    scene = build_scene(workload, ppc, TARGET_CAP)
    rule = RadianceConvergence(TARGET, minimum_rounds=32, check_every=1, consecutive_checks=1)
    backend = CUDA(device=device, seed=seed, guided=guided, roulette_scale=scale)

    with tempfile.TemporaryDirectory() as tmp:
        start = time.perf_counter()
        result = simulate(scene, backend, f"{tmp}/run.nc", convergence=rule)
        wall = time.perf_counter() - start
        receipt = json.loads(Path(f"{tmp}/run.run.json").read_text())

    relative = result.values["std_radiance"][..., 0, 0] / np.abs(result.values["radiance"][..., 0, 0])
    return {
        "seconds": wall,
        "status": receipt["status"],
        "rounds": int(receipt["completed_rounds"]),
        "max_relative_se": float(np.max(relative)),
        "median_relative_se": float(np.median(relative)),
        "scatters": int(receipt["scatters"]),
    }


def method_runs(workload, device, rank, guided, scale=None):
    """One method's time to target on every seed: medians of seconds and rounds, and of the
    variance x time merit 1 / (SE/|I|)^2 / seconds of the worst and of the median pixel."""

    runs = [time_to_target(workload, TARGET_PPC, device, seed + 1000 * rank, guided, scale) for seed in TARGET_SEEDS]
    median = lambda values: float(statistics.median(values))  # noqa: E731
    return {
        "seconds": median(r["seconds"] for r in runs),
        "rounds": median(r["rounds"] for r in runs),
        "worst_pixel_merit": median(1.0 / (r["max_relative_se"] ** 2 * r["seconds"]) for r in runs),
        "median_pixel_merit": median(1.0 / (r["median_relative_se"] ** 2 * r["seconds"]) for r in runs),
        "converged": all(r["status"] == "converged" for r in runs),
        "runs": runs,
    }


def end_to_end(workload, ppc, device, seed):
    """The e2e figure: ``simulate`` through the public API at the workload's own round size
    (host tables in, FP64 round statistics on the device, per-round pixel sums and the final
    statistics copied out, NetCDF product written), E2E_ROUNDS rounds."""

    import tempfile

    from monki import simulate
    from monki.execution import CUDA

    scene = build_scene(workload, ppc, E2E_ROUNDS)
    backend = CUDA(device=device, seed=seed)
    with tempfile.TemporaryDirectory() as tmp:
        start = time.perf_counter()
        simulate(scene, backend, f"{tmp}/run.nc")
        wall = time.perf_counter() - start
        receipt = json.loads(Path(f"{tmp}/run.run.json").read_text())
    nmat, nx, ny, nz, angles = scene.shape
    statistics_values = 3 * nmat * nx * ny * angles + (4 * nx * ny * nz * angles + 3 * nx * ny * angles if scene.save_path else 0)
    rounds = int(receipt["completed_rounds"])
    return {
        "seconds": wall,
        "rounds": rounds,
        "scatters": int(receipt["scatters"]),
        "scatters_per_s": receipt["scatters"] / wall,
        "h2d_bytes": int(scene.tables.nbytes + 32 * rounds),
        "d2h_bytes": int(rounds * nmat * 8 + statistics_values * 8),
    }


def learned_leg(workload, device, rank):
    """The learned importance: train the network on the device from analog importance tallies
    of the training family, turn its prediction for the workload into the per-cell weight
    window of guided transport, and time it to the target."""

    from monki.importance import LEARNED_GUIDE, learned_scale, train_model, training_scenes

    start = time.perf_counter()
    model, losses, rows = train_model(training_scenes(24), device=device)
    trained = time.perf_counter() - start
    fit_seconds = model.fit_seconds
    with model:
        scale = learned_scale(model, build_scene(workload, TARGET_PPC, 1))
    learned = method_runs(workload, device, rank, LEARNED_GUIDE, scale)
    learned["method"] = LEARNED_GUIDE.describe()
    # Dense-contraction figures of the network's training: FLOPs of the tcgen05 GEMMs per
    # step (forward 3 layers, backward weight and input gradients).
    flops = len(losses) * model.rows * 2 * (3 * (64 * 256 + 2 * 256 * 256) - 64 * 256)
    peaks_path = ROOT / "MEASURED_PEAKS.json"
    tensor_peak = json.loads(peaks_path.read_text()).get("bf16_tflops") if peaks_path.is_file() else 1900.0
    learned["training"] = {"seconds_with_pilots": trained, "fit_seconds": fit_seconds, "rows": rows,
                           "steps": len(losses), "batch": model.rows,
                           "loss_first": float(losses[:20].mean()), "loss_last": float(losses[-50:].mean()),
                           "gemm_tflops": flops / fit_seconds / 1e12,
                           "frac_of_bf16_peak": flops / fit_seconds / 1e12 / tensor_peak}
    return learned


# The reference's published time to AMF SE < 1 % (validation/README.md:230-233; Apple M4,
# end to end, median of three seeds, 8,000 photons per column, AMFConvergence defaults).
PUBLISHED_AMF = {
    "clear": {"metal_m4_s": 0.466, "cpu_m4_4_threads_s": 2.074},
    "layered_cloud": {"metal_m4_s": 26.160, "cpu_m4_4_threads_s": 232.839},
}


def reference_benchmark(device):
    """The reference's own benchmark on GB300: its clear and layered-cloud fixtures (prepared
    from its INPUT/DATA files, kept in tests/golden/), 8,000 photons per column, the
    AMFConvergence defaults, seeds 23274, 714103 and 19088743, one warm-up run, wall time of
    simulate() through the public API."""

    import tempfile
    from dataclasses import replace

    from monki import AMFConvergence, simulate
    from monki.execution import CUDA
    from monki.preparation import scene_from_arrays

    out = {}
    for name, published in PUBLISHED_AMF.items():
        scene = scene_from_arrays(np.load(ROOT / "tests" / "golden" / f"prepared_{name}.npz"))
        runs = []
        with tempfile.TemporaryDirectory() as tmp:
            simulate(replace(scene, rounds=2), CUDA(device=device), f"{tmp}/warmup.nc")
            for seed in (23274, 714103, 19088743):
                start = time.perf_counter()
                simulate(scene, CUDA(device=device, seed=seed), f"{tmp}/{seed}.nc", convergence=AMFConvergence())
                elapsed = time.perf_counter() - start
                receipt = json.loads(Path(f"{tmp}/{seed}.run.json").read_text())
                runs.append({"seed": seed, "seconds": elapsed, "status": receipt["status"],
                             "rounds": receipt["completed_rounds"], "scatters": receipt["scatters"]})
        median = statistics.median(r["seconds"] for r in runs)
        out[name] = {"median_s": median, "runs": runs, **published,
                     "speedup_vs_metal_m4": published["metal_m4_s"] / median,
                     "speedup_vs_cpu_m4": published["cpu_m4_4_threads_s"] / median}
    return out


def batched_scenes(device, scale):
    """The batched workload: 64 seeded scenes of uneven size (grids 8-128 columns a side,
    20-60 layers, log-uniform photon budgets scaled by ``scale``, lognormal cloud fields),
    one round each. Persistent: every scene in one multi-scene launch sequence (one shared
    photon pool; graph-replayed batches), after one warm-up run. Beside it, the scenes as
    concurrent sessions from four host threads with launch shapes from the autotuner
    (tuned once per size class), and one after another in their own sessions (default
    launch options), the way a caller without the batched API would run them."""

    import monki.scenes as scenes
    from monki.batched import run_batched, run_persistent
    from monki.tuning import autotune

    batch = [scenes.batched_scene(seed, photons_scale=scale) for seed in range(64)]
    run_persistent(batch[:8], device=device)  # warm-up: module load, graph instantiation
    _, persistent = run_persistent(batch, device=device)

    def size_class(scene):
        _, nx, ny, _, _ = scene.shape
        photons = scene.photons_per_column * nx * ny
        return 0 if photons < 1 << 20 else (1 if photons < 8 << 20 else 2)

    tuned = {}
    for scene in batch:
        tuned.setdefault(size_class(scene), autotune(scene, device=device))
    _, sessions = run_batched(batch, device=device, concurrency=4, tune=lambda s: tuned[size_class(s)].options(),
                              persistent=False)
    sessions["tuned"] = {str(k): v.options() for k, v in tuned.items()}
    _, one_at_a_time = run_batched(batch, device=device, concurrency=1, persistent=False)
    return {"photons_scale": scale, "persistent": persistent, "concurrent_sessions": sessions,
            "one_at_a_time": one_at_a_time}


def main():
    parser = argparse.ArgumentParser()
    parser.add_argument("--gpus", type=int, default=1)
    parser.add_argument("--steps", type=int, default=8)
    parser.add_argument("--warmup", type=int, default=3)
    parser.add_argument("--impl", default="gb300", choices=("gb300", "reference"))
    parser.add_argument("--workload", default="box", choices=tuple(WORKLOADS))
    parser.add_argument("--no-cpu-baseline", action="store_true")
    parser.add_argument("--no-target", action="store_true", help="skip the time-to-target runs")
    parser.add_argument("--no-learned", action="store_true", help="skip the learned-importance run")
    parser.add_argument("--no-batched", action="store_true", help="skip the batched-scenes run")
    parser.add_argument("--no-reference-benchmark", action="store_true",
                        help="skip the reference's time-to-AMF-precision benchmark")
    parser.add_argument("--batched-scale", type=float, default=0.05,
                        help="photon budgets of the batched scenes, as a fraction of the workload's")
    parser.add_argument("--photons-per-column", type=int, default=0)
    args = parser.parse_args()

    if args.warmup < 3:
        parser.error("at least 3 warm-up steps are required")

    if args.impl == "reference":
        return reference_arm(args)

    import torch

    from monki.execution import native as binding

    world, rank, local = distributed()
    torch.cuda.set_device(local)

    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl")

    def barrier():
        if world > 1:
            torch.distributed.barrier()

        torch.cuda.synchronize()

    _, default_ppc, workload = WORKLOADS[args.workload]
    ppc = args.photons_per_column or default_ppc
    scene = build_scene(args.workload, ppc, args.warmup + args.steps)
    nmat, nx, ny, nz, angles = scene.shape
    per_round = ppc * nx * ny
    native = binding.load()
    tables = np.ascontiguousarray(scene.tables)
    err = ctypes.create_string_buffer(4096)
    capacity = max(args.steps, args.warmup)  # every group has at most this many rounds
    handle = native.monki_cuda_create(
        local, tables.ctypes.data_as(binding.F64P), tables.size, capacity, b"precision=fp32", err, len(err)
    )

    if not handle:
        raise RuntimeError(err.value.decode())

    tally_count = int(native.monki_cuda_tally_count(handle))
    out = np.zeros(tally_count * capacity)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=f"cuda:{local}")
    timing = (ctypes.c_float * 2)()
    counters_before = (ctypes.c_uint64 * 6)()
    counters_after = (ctypes.c_uint64 * 6)()

    def group(start, rounds, profile=0):
        """One round group in one dispatch, as CUDA.run_batches schedules it (iteration
        batches replayed as CUDA graphs); ``profile`` adds per-stage event timing instead.
        Ranks run disjoint rounds (offset 100000 per rank)."""

        controls = (ctypes.c_uint32 * 8)(
            per_round * rounds, 0, first_round(rank, start), 0, 100000, profile, per_round, rounds
        )

        if native.monki_cuda_run(handle, controls, out.ctypes.data_as(binding.F64P), err, len(err)):
            raise RuntimeError(err.value.decode())

        native.monki_cuda_last_timing(handle, timing)
        return timing[0], timing[1]

    # Warm-up: W rounds, untimed.
    flush.zero_()
    torch.cuda.synchronize()
    group(1, args.warmup)
    native.monki_cuda_counters(handle, counters_before)
    flush.zero_()  # 256 MiB write: the timed group starts with a cold L2
    barrier()

    with Clocks(local) as clocks:
        wall = time.perf_counter()
        kernel_ms, run_ms = group(args.warmup + 1, args.steps)
        barrier()
        wall = time.perf_counter() - wall

    native.monki_cuda_counters(handle, counters_after)
    delta = [int(a) - int(b) for a, b in zip(counters_after, counters_before, strict=True)]
    scatters, visits_fp, visits_det, updates, photons, launches = delta
    # Per-stage timing for the roofline: a separate group of the same size with CUDA events
    # around every kernel (no graphs); its counters give the per-launch work.
    profiled_before = (ctypes.c_uint64 * 6)()
    profiled_after = (ctypes.c_uint64 * 6)()
    native.monki_cuda_counters(handle, profiled_before)
    flush.zero_()
    torch.cuda.synchronize()
    group(args.warmup + args.steps + 1, args.steps, profile=1)
    native.monki_cuda_counters(handle, profiled_after)
    stage_ms = (ctypes.c_double * 3)()
    stage_launches = (ctypes.c_uint64 * 3)()
    native.monki_cuda_stage_timing(handle, stage_ms, stage_launches)
    p_scatters, p_visits_fp, p_visits_det, p_updates, _, _ = (
        int(a) - int(b) for a, b in zip(profiled_after, profiled_before, strict=True)
    )
    device_seconds = run_ms / 1e3

    if world > 1:
        device_seconds, total_scatters = combine_ranks(device_seconds, scatters, f"cuda:{local}")
    else:
        total_scatters = float(scatters)

    native.monki_cuda_close(handle)
    value = total_scatters / device_seconds
    # Roofline per wavefront kernel: algorithmic bytes per launch over the event-timed
    # launch duration; the line reports the kernel with the largest share of device time.
    #   step     (scenes without layer paths) each event's list entry, its state read once
    #            and written once, its new queue entry, 16 B per free-path cell visit
    #   transit  each event's state read and written and its queue entry, 16 B per
    #            free-path cell visit
    #   peel     each event's state, 16 B per detector-ray cell visit, 32 B per tally atomic
    #   scatter  each event's queue entry and state read and written
    peak, peak_kind = peaks()
    stage_total = max(sum(stage_ms), 1e-9)
    fused = not scene.save_path  # the session's default: fused step unless the scene has layer paths
    names = ("step", "peel") if fused else ("transit", "peel", "scatter")
    stage_share = {name: stage_ms[q] / stage_total for q, name in enumerate(names)}
    algorithmic = {
        "step": STEP_EVENT_BYTES * p_scatters + CELL_BYTES * p_visits_fp,
        "transit": TRANSIT_EVENT_BYTES * p_scatters + CELL_BYTES * p_visits_fp,
        "peel": STATE_BYTES * p_scatters + CELL_BYTES * p_visits_det + TALLY_BYTES * p_updates,
        "scatter": SCATTER_EVENT_BYTES * p_scatters,
    }
    kernels = {}
    for q, name in enumerate(names):
        launches_q = max(int(stage_launches[q]), 1)
        seconds = stage_ms[q] / 1e3 / launches_q
        per_launch = algorithmic[name] / launches_q
        kernels[name] = {
            "algorithmic_bytes_per_launch": per_launch,
            "launch_ms": seconds * 1e3,
            "launches": launches_q,
            "achieved_gbs": per_launch / seconds / 1e9,
            "frac": per_launch / seconds / 1e9 / peak,
            "traffic": recorded_traffic(args.workload, name, per_launch),
            "share": stage_share[name],
        }
    dominant = max(names, key=lambda name: stage_share[name])

    # Everything after the timed region is reported, never fatal: a leg that raises is
    # recorded as {"error": ...} in the line, so no extra can erase the measurement.
    def attempt(leg):
        try:
            return leg()
        except Exception as exc:  # noqa: BLE001 - reported in the JSON line
            return {"error": f"{type(exc).__name__}: {exc}"[:800]}

    # Time to the precision target through the public API, analog then guided, on every
    # rank (independent seeds); the analog run is also the end-to-end throughput.
    from monki import Guided

    e2e = attempt(lambda: end_to_end(args.workload, ppc, local, 23274 + rank))
    target = None
    if not args.no_target:
        barrier()
        target = {"analog": attempt(lambda: method_runs(args.workload, local, rank, None)),
                  "guided": attempt(lambda: method_runs(args.workload, local, rank, Guided(*GUIDED)))}

        if not args.no_learned:
            target["guided_learned"] = attempt(lambda: learned_leg(args.workload, local, rank))

    if rank != 0:
        if world > 1:
            torch.distributed.destroy_process_group()

        return 0

    line = {
        "metric": METRIC,
        "value": value,
        "unit": UNIT,
        "n_gpus": world,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": device_seconds / args.steps * 1e3,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": {
            "workload": workload,
            "photons_per_step": per_round,
            "scatters_per_step": scatters / args.steps,
            "l2": "flushed before the timed round group by a 256 MiB device write; the scene "
            "tables (< 2 MB) stay L2-resident by design",
            "parallelism": f"{world} independent round streams" if world > 1 else "1 GPU",
            "wall_s": wall,
        },
        "roofline": {
            "bound": "hbm",
            "kernel": f"wf_{dominant}",
            "achieved": kernels[dominant]["achieved_gbs"],
            "peak": peak,
            "unit": "GB/s",
            "frac": kernels[dominant]["frac"],
            "traffic": kernels[dominant]["traffic"],
            "peak_source": peak_kind,
            "algorithmic_bytes_per_launch": kernels[dominant]["algorithmic_bytes_per_launch"],
            "launch_ms": kernels[dominant]["launch_ms"],
            "launches": kernels[dominant]["launches"],
            "stage_share": stage_share,
            "kernels": kernels,
        },
        "gpu_launches": launches,
        "clocks": clocks.summary(),
    }

    if target is not None:
        summary = {"target": f"SE/|I| < {TARGET:g} in every pixel and view, checked every round from round 32",
                   "photons_per_column": TARGET_PPC, "seeds": list(TARGET_SEEDS),
                   "guided_method": Guided(*GUIDED).describe(), **target}
        plain = target["analog"]
        for name in ("guided", "guided_learned"):
            other = target.get(name, {})
            if "seconds" in plain and "seconds" in other:
                summary[f"{name}_speedup"] = plain["seconds"] / other["seconds"]
                summary[f"{name}_worst_pixel_gain"] = other["worst_pixel_merit"] / plain["worst_pixel_merit"]
                summary[f"{name}_median_pixel_gain"] = other["median_pixel_merit"] / plain["median_pixel_merit"]
        if "worst_pixel_merit" in target.get("guided_learned", {}) and "worst_pixel_merit" in target["guided"]:
            summary["learned_over_constant_worst_pixel"] = (target["guided_learned"]["worst_pixel_merit"]
                                                            / target["guided"]["worst_pixel_merit"])
        line["time_to_target"] = summary
    if "scatters_per_s" in e2e:
        line["e2e"] = {
            "value": e2e["scatters_per_s"] * world,
            "unit": UNIT,
            "h2d_bytes_per_step": e2e["h2d_bytes"] / e2e["rounds"],
            "d2h_bytes_per_step": e2e["d2h_bytes"] / e2e["rounds"],
            "wall_s": e2e["seconds"],
            "rounds": e2e["rounds"],
            "note": "simulate() with CUDA() on the workload at its own round size: table upload, FP64 round "
            "statistics on the device, per-round pixel sums and the final statistics copied to the host, NetCDF "
            "product written",
        }
    else:
        line["e2e"] = e2e

    if not args.no_cpu_baseline:
        line["cpu_baseline"] = attempt(lambda: cpu_baseline(build_scene(args.workload, ppc, 1)))

    if not args.no_batched:
        line["batched"] = attempt(lambda: batched_scenes(local, args.batched_scale))

    if not args.no_reference_benchmark:
        line["reference_benchmark"] = attempt(lambda: reference_benchmark(local))

    if not args.no_target:
        # FP32 bias of the product transport against the FP64 build, per Stokes component.
        from monki.precision import fp32_bias

        line["fp32_bias"] = attempt(lambda: fp32_bias(build_scene(args.workload, 2000, 8), rounds=8,
                                                      photons_per_column=2000, device=local))

    print(json.dumps(line))

    if world > 1:
        torch.distributed.destroy_process_group()

    return 0


if __name__ == "__main__":
    sys.exit(main())
