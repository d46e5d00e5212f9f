"""Benchmark of the SPH substep on GB300 (one JSON line on stdout, rank 0).

A "step" is one substep (sph_simulation::simulate_single_frame) over the
whole scene. Default workload: the 1,048,576-particle dam break (128 x 128 x 64
lattice at spacing h/2 = 1/128 m in the left quarter of a 4 x 2 x 2 m box, 12
triangles), synthetic and seeded.

  value     particle-steps/s with the particles resident in HBM; each timed
            step is bracketed by CUDA events on the engine's stream, and a
            256 MiB buffer is written between steps (outside the events) so
            every step starts with a cold L2.
  e2e       the same metric through the public C ABI with HOST buffers: each
            step uploads the 80-byte particle AoS from pinned memory, runs
            the substep and downloads the AoS (the reference's per-substep
            transfer pattern, sph_simulation.cpp:195-197, 339-341); the
            engine's unpacking and packing kernels read and write the pinned
            records in place over the host link.
  long_run  the same K substeps as one uninterrupted clsph_gpu_step(K) (graph
            replays of 16 substeps, no flush), beside the headline value.
  roofline  the dominant kernel: algorithmic bytes per launch / its mean
            CUDA-event duration, against the measured HBM copy bandwidth.
  cpu_baseline  the CPU oracle (the restatement of the reference's substep,
            OpenMP over particles, all host threads) on a bounded sample.

--impl reference times the reference's CPU implementation of the path (the
oracle port; the OpenCL CPU device is unavailable on these hosts) on the same
workload at full size, all host threads, the same --steps and --warmup, and
prints the same `config`. Only a workload whose full-size substeps would take
longer than REFERENCE_BUDGET_S in all (the pour's brute-force collision over
131,072 triangles) is timed on a 65,536-particle sample, and its config then
says so.

Multi-GPU: a single scene does not shard (no halo exchange is built), so N
ranks run N independent replicas of it (weak scaling); the batched workload
splits its scenes over the ranks by particle count (strong scaling). There is
no collective on the data path, only the barrier and the timing reductions.
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

# algorithmic HBM bytes per particle for each kernel (compulsory traffic of
# its inputs and outputs, neighbour re-reads excluded)
ALG_BYTES_PER_PARTICLE = {
    "keys": 16 + 4,                 # read position, write key
    "radix_sort": 3 * 16,           # read key+slot, write key+slot, three passes
    "gather": 4 + 48 + 48 + 8,      # read slot, read + write state, ids
    "density": 16 + 8,              # read position, write density + pressure
    "forces": 32 + 8 + 16,          # read position, velocity, density, pressure; write acceleration
    "advect": 48 + 48,              # read position, half-step velocity, acceleration; write state
}
STEP_ALG_BYTES = 232  # per particle-substep: key read 16 + sort scatter 96 + density 20 + forces/integrate 100
# FP32 operations of the exact pair arithmetic, one per IEEE add, multiply,
# divide or square root (the kernels use no FMAs there): a density pair
# (forces.cl:33-36) and a force pair (forces.cl:67-97), and per particle the
# Tait pressure with its quotients (sph.cl:36-39) and the acceleration
# (forces.cl:103-109, sph.cl:53-58)
FLOP_DENSITY_PAIR = 16
FLOP_FORCE_PAIR = 65
FLOP_PER_PARTICLE = 30
# FP32 peak of a GB300 at its maximum SM clock (2070 MHz): 152 SMs x 128
# lanes x 2 (an FMA counted as two operations) = 80.5 TFLOP/s
FP32_PEAK_TFLOPS = 152 * 128 * 2 * 2070e6 / 1e12


def mean_pairs(scene, particles) -> float | None:
    """Mean number of particles within h of a particle (itself included)
    in the given state: the pairs the exact arithmetic evaluates."""
    try:
        from scipy.spatial import cKDTree
    except ImportError:
        return None
    parts = scene.scenes if isinstance(scene, Batch) else [scene]
    total, first = 0, 0
    for s in parts:
        n = len(s.particles)
        pos = np.asarray(particles["position"][first:first + n, :3], dtype=np.float64)
        h = float(s.params["h"])
        total += int(cKDTree(pos).query_pairs(h, output_type="ndarray").shape[0]) * 2 + n
        first += n
    return total / max(first, 1)

def _w():
    return __import__("libclsph_gb300.workloads", fromlist=["x"])


WORKLOADS = {
    "dam_break_1m": lambda: _w().dam_break_1m(),
    "dam_break_32k": lambda: _w().dam_break_32k(),
    "pour_4m": lambda: _w().pour(),
    "batched_256": lambda: _w().batched_dam_breaks(256),
}


class Batch:
    """A list of scenes run by one batched handle."""

    def __init__(self, scenes):
        self.scenes = scenes
        self.name = f"batched_{len(scenes)}_dam_breaks"
        self.particles = np.concatenate([s.particles for s in scenes])
        self.params = scenes[0].params
        self.mesh = scenes[0].mesh
        self.info = {"scenes": len(scenes), "n_min": min(s.n for s in scenes),
                     "n_max": max(s.n for s in scenes)}

    @property
    def n(self):
        return len(self.particles)


def load_workload(name, world: int = 1, rank: int = 0):
    """The workload of this rank: a replica of a single scene, or this rank's
    share of a batch's scenes."""
    w = WORKLOADS[name]()
    if isinstance(w, list):
        if world > 1:
            w = [w[k] for k in partition_scenes([s.n for s in w], world)[rank]]
        return Batch(w)
    return w


def make_solver(scene):
    from libclsph_gb300.gpu import GpuSolver

    if isinstance(scene, Batch):
        sc = scene.scenes
        return GpuSolver.batched([s.params for s in sc], [s.terms for s in sc], [s.n for s in sc],
                                 [s.mesh for s in sc])
    return GpuSolver(scene.params, scene.terms, scene.n, scene.mesh)


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def measured_peaks() -> tuple[float, str]:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return float(json.loads(p.read_text())["hbm_gbs"]), "measured"
        except Exception:
            pass
    return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clock / throttle samples during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.path = None

    def __enter__(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200", "-f", self.path],
                stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
            time.sleep(0.3)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            time.sleep(0.25)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self) -> dict:
        if not self.path or not Path(self.path).exists():
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in Path(self.path).read_text().splitlines():
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower() == "active":
                    reasons.add(name)
        Path(self.path).unlink(missing_ok=True)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "samples": len(sm),
                "reasons": sorted(reasons)}


def dist_setup(backend: str | None = None):
    """Rank, world size and local rank from the torchrun environment; one
    process per GPU over NCCL (gloo on hosts without CUDA). The ranks only
    meet for the barrier and the timing reductions: each one runs its own
    replica (or its own share of a batch's scenes) with no collective on the
    data path."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch
        import torch.distributed as dist

        if backend is None:
            backend = "nccl" if torch.cuda.is_available() else "gloo"
        if not dist.is_initialized():
            dist.init_process_group(backend)
    return world, rank, local


def _reduce(x: float, world: int, op: str) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist

    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], device=dev, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX if op == "max" else dist.ReduceOp.SUM)
    return float(t.item())


def max_over_ranks(x: float, world: int) -> float:
    return _reduce(x, world, "max")


def sum_over_ranks(x: float, world: int) -> float:
    return _reduce(x, world, "sum")


def partition_scenes(sizes, world: int) -> list[list[int]]:
    """Scenes of a batch split over ranks by particle count (longest first to
    the least-loaded rank); every scene on exactly one rank."""
    loads = [0] * world
    parts: list[list[int]] = [[] for _ in range(world)]
    for k in sorted(range(len(sizes)), key=lambda k: (-sizes[k], k)):
        r = min(range(world), key=lambda q: (loads[q], q))
        parts[r].append(k)
        loads[r] += sizes[k]
    return [sorted(p) for p in parts]


def barrier(world: int) -> None:
    if world > 1:
        import torch.distributed as dist

        dist.barrier()


def cpu_sample_scene(scene, count: int):
    """The first `count` lattice particles of the scene: same spacing, mass,
    h and mesh, so per-particle work matches the full scene."""
    from libclsph_gb300.workloads import Scene

    params = np.array(scene.params).copy()
    params["particles_count"] = count
    return Scene(scene.name + f"_sample{count}", params, scene.terms,
                 scene.particles[:count].copy(), scene.mesh, scene.steps, dict(scene.info))


def cpu_baseline(scene, target_s: float = 12.0) -> dict:
    from oracle import Oracle

    o = Oracle()
    threads = os.cpu_count() or 1
    if isinstance(scene, Batch):  # scenes one after another, as many as the budget allows
        done = 0
        t0 = time.perf_counter()
        k = 0
        while time.perf_counter() - t0 < target_s and k < len(scene.scenes):
            sc = scene.scenes[k]
            o.run(sc.params, sc.terms, sc.particles, 1, sc.mesh, threads=threads)
            done += sc.n
            k += 1
        dt = time.perf_counter() - t0
        return {"value": done / dt, "unit": "particle-steps/s", "cores": threads, "kind": "port",
                "sample": f"one substep of each of the first {k} of {len(scene.scenes)} scenes "
                          f"({done} particle-steps, {dt:.1f} s, OpenMP over particles)"}
    n = scene.n
    what = f"the full {n}-particle workload"
    if n > 65536:
        # when one substep of the whole scene would exceed the budget (the
        # pour's 131k-triangle brute-force collision), time a particle sample
        probe = cpu_sample_scene(scene, 65536)
        t0 = time.perf_counter()
        o.run(probe.params, probe.terms, probe.particles, 1, probe.mesh, threads=threads)
        if (time.perf_counter() - t0) * n / 65536 > target_s:
            scene, n = probe, 65536
            what = "a 65536-particle sample (same spacing, mass, h and mesh)"
    steps = 0
    t0 = time.perf_counter()
    cur = scene.particles
    while True:
        cur = o.run(scene.params, scene.terms, cur, 1, scene.mesh, threads=threads)
        steps += 1
        if time.perf_counter() - t0 >= target_s or steps >= 20:
            break
    dt = time.perf_counter() - t0
    return {"value": n * steps / dt, "unit": "particle-steps/s", "cores": threads, "kind": "port",
            "sample": f"{steps} substeps of {what} from its initial state "
                      f"({dt:.1f} s, OpenMP over particles)"}


REFERENCE_BUDGET_S = 300.0  # longest full-size reference run (warm-up + timed substeps)


def workload_config(scene, args, n_particles: int | None = None) -> dict:
    """The `config` object of both arms' JSON lines (identical for the same
    workload and flags)."""
    return {
        "workload": scene.name,
        "n_particles": scene.n if n_particles is None else n_particles,
        "lattice": scene.info.get("lattice"),
        "box_m": scene.info.get("box"),
        "h_m": scene.info.get("h"),
        "scenes": scene.info.get("scenes", 1),
        "faces": len(scene.mesh["indices"]) // 3,
        "l2": ("inputs larger than L2: a substep moves about 460 B per particle through DRAM "
               "(neighbour lists, records, state; profiles/dram_bytes_per_particle.json); the GPU "
               "arm also writes a 256 MiB buffer before every timed launch, outside its events")
              if not args.no_flush else
              "inputs larger than L2: a substep moves about 460 B per particle through DRAM; no flush",
    }


def run_reference(args, world, rank) -> None:
    if rank != 0:
        return
    from oracle import Oracle

    scene = load_workload(args.workload)
    o = Oracle()
    threads = os.cpu_count() or 1

    def make_units(full: bool):
        if full:
            return scene.scenes if isinstance(scene, Batch) else [scene]
        if isinstance(scene, Batch):  # the first scenes, up to ~65k particles
            take, tot = [], 0
            for sc in scene.scenes:
                if tot >= 65536:
                    break
                take.append(sc)
                tot += sc.n
            return take
        return [cpu_sample_scene(scene, min(65536, scene.n))]

    units = make_units(True)
    cur = [u.particles for u in units]

    def one_step():
        for k, u in enumerate(units):
            cur[k] = o.run(u.params, u.terms, cur[k], 1, u.mesh, threads=threads)

    # the first warm-up substep at full size decides whether the whole run fits
    t0 = time.perf_counter()
    one_step()
    first_s = time.perf_counter() - t0
    full = first_s * (args.steps + args.warmup - 1) <= REFERENCE_BUDGET_S
    if not full:
        units = make_units(False)
        cur = [u.particles for u in units]
        one_step()
    for _ in range(args.warmup - 1):
        one_step()
    n_done = sum(u.n for u in units)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        one_step()
    dt = time.perf_counter() - t0
    value = n_done * args.steps / dt
    what = (f"all {scene.n} particles per substep (the full workload)" if full else
            f"{n_done} of the {scene.n} particles per substep (same spacing, mass, h, mesh): the full "
            f"substep takes {first_s:.0f} s here")
    line = {
        "impl": "reference", "metric": "particle-steps/s", "value": value,
        "unit": "particle-steps/s", "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1e3 * dt / args.steps, "higher_is_better": True,
        "scaling": "strong" if isinstance(scene, Batch) else "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": workload_config(scene, args, None if full else n_done),
        "cpu_baseline": {"value": value, "unit": "particle-steps/s", "cores": threads, "kind": "port",
                         "sample": f"{what}; {args.steps} timed substeps after {args.warmup} warm-up "
                                   f"substeps, OpenMP over particles on every host thread; the "
                                   f"reference's OpenCL CPU device has no platform on these hosts, so "
                                   f"the oracle restatement of its kernels runs instead"},
        "e2e": {"value": value, "unit": "particle-steps/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_mlp_rows(args) -> None:
    """`--workload mlp_1m_rows`: the learned stepper's fused MLP inference
    kernels alone on 1,048,576 random standardised feature rows (random
    weights): CUDA events around each launch after the warm-up launches, the
    tcgen05 kernel (clsph_mlp_forward) and the mma.sync cross-check
    (clsph_mlp_forward_mma_sync). FLOPs count 2 per multiply-add of the three
    layers, 2 * rows * (32*256 + 256*256 + 256*4); the roofline is the
    measured BF16 tensor peak."""
    import torch

    from libclsph_gb300 import learned as Lm

    rows = 1 << 20
    torch.cuda.set_device(0)
    blob = np.zeros(Lm.BLOB, np.float32)
    rng = np.random.default_rng(0)
    blob[:Lm.N_PARAMS] = rng.normal(0, 0.05, Lm.N_PARAMS)
    blob[Lm.OFF_XSIGMA:Lm.OFF_YMU] = 1
    blob[Lm.OFF_YSIGMA:] = 1
    net = Lm.Mlp(blob=blob)
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(rows, Lm.N_FEATURES, device="cuda", generator=g).to(torch.bfloat16)
    y = torch.empty(rows, Lm.N_OUTPUTS, device="cuda")
    flops = 2.0 * rows * (32 * 256 + 256 * 256 + 256 * 4)
    peaks = ROOT / "MEASURED_PEAKS.json"
    peak = json.loads(peaks.read_text()).get("bf16_tflops") if peaks.exists() else None
    peak_kind = "measured" if peak else "fallback"
    peak = peak or 1900.0
    out = {}
    for name, fn in (("tcgen05", net.forward), ("mma_sync", net.forward_mma_sync)):
        for _ in range(args.warmup):
            fn(x.data_ptr(), rows, y.data_ptr())
        torch.cuda.synchronize()
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
              for _ in range(args.steps)]
        for a, b in ev:
            a.record()
            fn(x.data_ptr(), rows, y.data_ptr())
            b.record()
        torch.cuda.synchronize()
        ms = sum(a.elapsed_time(b) for a, b in ev) / len(ev)
        out[name] = {"ms": ms, "tflops": flops / ms / 1e9}
    status = net.status()
    net.close()
    tc = out["tcgen05"]
    line = {
        "metric": "TFLOP/s", "value": tc["tflops"], "unit": "TFLOP/s", "n_gpus": 1,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": tc["ms"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "bf16 (fp32 accumulation)", "data": "synthetic",
        "config": {"workload": "mlp_1m_rows", "rows": rows, "layers": "32-256-256-4, GELU",
                   "l2": "64 MB of feature rows per launch, no flush"},
        "roofline": {"bound": "tensor", "kernel": "k_mlp_tc", "achieved": tc["tflops"], "peak": peak,
                     "peak_kind": peak_kind, "unit": "TFLOP/s", "frac": tc["tflops"] / peak,
                     "traffic": None},
        "mma_sync": out["mma_sync"], "device_status": status, "gpu_launches": 2 * (args.steps + args.warmup),
    }
    print(json.dumps(line), flush=True)


def learned_evaluation(scene, solver) -> dict | None:
    """Plain vs learned 4x-dt over the time of 2000 plain substeps, with the 1 %
    density check and without it (weights from
    libclsph_gb300/weights/stepper_4dt.npz; skipped when absent)."""
    from libclsph_gb300 import learned as Lm
    from libclsph_gb300.stepper_eval import evaluate

    path = Lm.default_weights_path()
    if not path.exists():
        return {"skipped": f"no weights at {path.relative_to(ROOT)}"}
    import torch

    mlp = Lm.Mlp.load(path)
    solver.set_graph(False)
    torch.cuda.synchronize()
    r = evaluate(scene, mlp, plain_substeps=2000, dt_mult=4, checkpoints=10, threshold=0.01)
    # the same network without the density check: every step learned
    r_free = evaluate(scene, mlp, plain_substeps=2000, dt_mult=4, checkpoints=10, check=False)
    mlp.close()
    keep = ("plain_sim_s_per_s", "learned_sim_s_per_s", "speedup", "fallback_fraction", "accepted_steps",
            "rejected_steps", "check_deviation_mean", "check_deviation_max", "density_dev",
            "density_dev_max", "density_dev_pop", "density_dev_particle", "rho_dev_plain",
            "rho_dev_learned", "pos_rms_h_final", "pos_rms_chaos_h_final", "density_dev_chaos", "threshold", "dt_mult",
            "plain_substeps", "learned_steps", "sim_time_s")
    out = {k: r[k] for k in keep}
    out["curve_t"] = [c["t"] for c in r["curve"]]
    out["curve_density_dev"] = [c["density_dev"] for c in r["curve"]]
    out["curve_pos_rms_h"] = [c["pos_rms_h"] for c in r["curve"]]
    out["curve_pos_rms_chaos_h"] = [c["pos_rms_chaos_h"] for c in r["curve"]]
    out["curve_ke_plain"] = [c["ke_plain"] for c in r["curve"]]
    out["curve_ke_learned"] = [c["ke_learned"] for c in r["curve"]]
    out["no_check"] = {k: r_free[k] for k in ("learned_sim_s_per_s", "plain_sim_s_per_s", "speedup",
                                              "density_dev", "density_dev_max", "pos_rms_h_final")}
    return out


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--workload", default="dam_break_1m", choices=sorted(WORKLOADS) + ["mlp_1m_rows"])
    ap.add_argument("--e2e-steps", type=int, default=20)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-flush", action="store_true")
    ap.add_argument("--no-graph", action="store_true", help="launch every kernel instead of replaying a CUDA graph")
    ap.add_argument("--no-autotune", action="store_true")
    ap.add_argument("--no-learned", action="store_true",
                    help="skip the learned 4x-dt stepper's evaluation on the 1M dam break")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    # the reference arm runs on the host cores only: its ranks meet over gloo
    world, rank, local = dist_setup("gloo" if args.impl == "reference" else None)
    if args.impl == "reference":
        run_reference(args, world, rank)
        barrier(world)
        return
    if args.workload == "mlp_1m_rows":
        run_mlp_rows(args)
        return

    import torch

    from libclsph_gb300.gpu import GpuSolver, load_library
    from libclsph_gb300.layout import PARTICLE

    torch.cuda.set_device(local)
    load_library()
    scene = load_workload(args.workload, world, rank)
    n = scene.n
    log(f"[rank {rank}] {scene.name}: n={n}")
    stream = torch.cuda.Stream()
    solver = make_solver(scene)
    solver.set_stream(stream.cuda_stream)
    solver.upload(scene.particles)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    tuning = None
    if not args.no_autotune:
        tuning = solver.autotune(3)
        log(tuning)
    unit = 1 if args.no_graph else 2  # substeps per timed launch unit
    solver.set_graph(not args.no_graph)
    args.steps = max(unit, args.steps - args.steps % unit)

    for _ in range(max(1, args.warmup // unit)):
        solver.step(unit)
    flags = solver.sync()

    # ---- timed region: K substeps on resident particles
    solver.set_profiling(True)
    launches0 = solver.counters()["launches"]
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(args.steps // unit)]
    barrier(world)
    torch.cuda.synchronize()
    with ClockSampler(local) as clocks:
        wall0 = time.perf_counter()
        with torch.cuda.stream(stream):
            for k in range(args.steps // unit):
                if not args.no_flush:
                    flush.fill_(float(k))
                ev[k][0].record(stream)
                solver.step(unit)
                ev[k][1].record(stream)
        torch.cuda.synchronize()
        wall = time.perf_counter() - wall0
    barrier(world)
    step_ms = [a.elapsed_time(b) for a, b in ev]
    flags |= solver.sync()
    launches = solver.counters()["launches"] - launches0
    solver.set_profiling(False)
    # per-kernel durations: a separate pass with events around every kernel
    # (graph replay has no per-kernel events), same state, no flush
    solver.set_profiling(True)
    with torch.cuda.stream(stream):
        for _ in range(min(args.steps, 40)):
            solver.step(1)
    torch.cuda.synchronize()
    prof_steps = min(args.steps, 40)
    ktimes = solver.kernel_times()
    solver.set_profiling(False)
    device_s = sum(step_ms) / 1e3
    device_s_max = max_over_ranks(device_s, world)
    total_particles = sum_over_ranks(float(n), world)
    value = total_particles * args.steps / device_s_max

    # ---- the same K substeps as one uninterrupted run (what a long
    # simulation sees: 16-substep graph replays, no flush; inputs larger
    # than L2), reported beside the headline value, not instead of it
    long_run = None
    if not args.no_graph:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        barrier(world)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            e0.record(stream)
            solver.step(args.steps)
            e1.record(stream)
        torch.cuda.synchronize()
        long_s = max_over_ranks(e0.elapsed_time(e1) / 1e3, world)
        flags |= solver.sync()
        long_run = {"value": total_particles * args.steps / long_s, "unit": "particle-steps/s",
                    "substeps": args.steps, "ms_per_step": 1e3 * long_s / args.steps,
                    "how": "one CUDA-event pair around clsph_gpu_step(K): graph replays of 16 substeps, no L2 flush"}

    # ---- end to end through the C ABI with host buffers (one substep per transfer pair)
    host = torch.empty(n * PARTICLE.itemsize, dtype=torch.uint8, pin_memory=True)
    aos = host.numpy().view(PARTICLE)
    aos[:] = solver.download()
    barrier(world)
    t0 = time.perf_counter()
    for _ in range(args.e2e_steps):
        solver.upload(aos)
        solver.step(1)
        solver.download(aos)
    e2e_s = max_over_ranks(time.perf_counter() - t0, world)
    e2e_value = total_particles * args.e2e_steps / e2e_s
    flags |= solver.sync()

    # ---- roofline of the dominant kernel
    peak, peak_kind = measured_peaks()
    dom = max((k for k in ktimes if ktimes[k][1] > 0), key=lambda k: ktimes[k][0])
    dom_ms, dom_count = ktimes[dom]
    dom_mean_s = dom_ms / dom_count / 1e3
    alg_bytes = ALG_BYTES_PER_PARTICLE.get(dom, 0) * n
    achieved = alg_bytes / dom_mean_s / 1e9 if dom_mean_s > 0 else 0.0
    traffic = None
    tfile = ROOT / "profiles" / "dram_bytes_per_particle.json"
    if tfile.exists():
        try:
            per = json.loads(tfile.read_text()).get(args.workload, {}).get(dom)
            traffic = per * n if per is not None else None
        except Exception:
            traffic = None
    step_achieved = STEP_ALG_BYTES * n * args.steps / device_s / 1e9
    # FP32 pipe: the exact pair arithmetic over the pairs of the final state
    pairs = mean_pairs(scene, aos)
    fp32 = None
    if pairs is not None:
        flop = (FLOP_DENSITY_PAIR + FLOP_FORCE_PAIR) * pairs + FLOP_PER_PARTICLE
        fp32_achieved = flop * value / 1e12
        fp32 = {"pairs_per_particle": pairs, "flop_per_particle_step": flop, "achieved_tflops": fp32_achieved,
                "peak_tflops": FP32_PEAK_TFLOPS, "frac": fp32_achieved / FP32_PEAK_TFLOPS,
                "how": "one FLOP per IEEE add, multiply, divide and square root of the exact density and force "
                       "pair arithmetic over the neighbour pairs of the final state; peak 152 SMs x 128 lanes x "
                       "2 x 2070 MHz"}

    # ---- learned 4x-dt stepper against the plain solver (the 1M dam break only)
    learned = None
    if not args.no_learned and args.workload == "dam_break_1m":
        learned = learned_evaluation(scene, solver)

    if rank != 0:
        return
    cpu = None
    if not args.no_cpu_baseline:
        try:
            cpu = cpu_baseline(scene)
        except Exception as e:  # an oracle failure must not hide the GPU number
            cpu = {"value": None, "unit": "particle-steps/s", "cores": os.cpu_count(),
                   "kind": "port", "sample": f"failed: {e}"}
    line = {
        "metric": "particle-steps/s",
        "value": value,
        "unit": "particle-steps/s",
        "n_gpus": args.gpus,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": 1e3 * device_s_max / args.steps,
        "higher_is_better": True,
        "scaling": "strong" if isinstance(scene, Batch) else "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": workload_config(scene, args),
        "timed_launch_substeps": unit,
        "sim_s_per_s": value / n * float(scene.params["time_delta"] * scene.params["simulation_scale"]),
        "wall_s_timed_region": wall,
        "roofline": {
            "bound": "hbm",
            "kernel": dom,
            "achieved": achieved,
            "peak": peak,
            "peak_kind": peak_kind,
            "unit": "GB/s",
            "frac": achieved / peak,
            "traffic": traffic,
            "alg_bytes_per_launch": alg_bytes,
            "mean_launch_ms": dom_mean_s * 1e3,
            "step_alg_GBps": step_achieved,
            "step_frac": step_achieved / peak,
            "fp32": fp32,
        },
        "kernel_ms_per_step": {k: v[0] / prof_steps for k, v in ktimes.items() if v[1]},
        "long_run": long_run,
        "launch": {"graph": not args.no_graph, "autotune": tuning.strip().splitlines()[-1] if tuning else None},
        "cpu_baseline": cpu,
        "e2e": {"value": e2e_value, "unit": "particle-steps/s",
                "h2d_bytes_per_step": n * PARTICLE.itemsize,
                "d2h_bytes_per_step": n * PARTICLE.itemsize, "steps": args.e2e_steps},
        "learned": learned,
        "gpu_launches": launches,
        "device_flags": flags,
        "clocks": clocks.summary(),
    }
    print(json.dumps(line), flush=True)
    solver.close()


if __name__ == "__main__":
    main()
