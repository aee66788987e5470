#!/usr/bin/env python
"""Benchmark of the CCpol23+(2025) force-evaluation hot path on B200.

A step is one evaluation of the hot path of the 512-water FS2+FS3 box (L = 24.84 A,
seeded synthetic configuration): Ewald self/intramolecular, real and reciprocal sums,
the induced-dipole solve with induction forces, FS2 and FS3 (SR/LR/blend).  The 2-body
term and the integrator are outside this path.  ns/day = steps/s x 0.0005 ps x 86400 / 1000
(dt = 0.5 fs).  Two forms are timed: FP64 and the mixed-precision form.  The headline value is
the faster end to end, the mixed form only if its relative force errors against the FP64 form
(site forces, per-molecule forces, torques) are all <= 1e-5; both are reported.

  python bench.py [--gpus N --steps K --warmup W] [--impl reference]

With --impl reference the CPU oracle (the reference's algorithm restated in C, the reference
itself being Fortran/MPI with no compiler on this image) runs the same step on all host
cores.  Multi-GPU runs are independent replicas (the path does not shard here): one seeded
box per rank, no collectives in the timed region.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "ns/day @512 H2O FS2+FS3: mixed vs FP64 GPU at rel force err <=1e-5; triples/s"
# the large-box configuration (bench.py --config c5_2048), reported with the same keys
METRIC_C5 = "ns/day @2048 H2O FS2+FS3: mixed vs FP64 GPU at rel force err <=1e-5; triples/s"
DT_PS = 0.0005
CONFIG = "c2_512"
# Algorithmic work of one FS3 site-triple evaluation (energy + gradient, one SR or LR
# representation), as the reference computes it: ~130 FLOP + 15 MUFU-class operations
# (6 exp, 3 sqrt, 6 reciprocals).  Counted as 145 floating-point operations.
FS3_FLOP_PER_SITE_TRIPLE = 145.0
# FP64 operations that FS3 by molecule pairs executes (k_fs3_pairs.cu), a DMMA counted as 512 with
# its zero padding.  A visit of the pair kernel, three per sum: 80 DMMA (40,960), the sums with a
# site 0 and the weights (8448 + 1728).  An energy sum: 80 DMMA (40,960), the contraction with the
# coefficients and the edges (40,344).  A triple has one sum, two in the blend region.  Work per
# molecule pair (tables, coefficients, forces) is not counted.
FS3_FLOP_PER_SUM = 3 * 51136.0 + 81304.0
# Precision forms the bench can time: context precision and options.  "mixed" is the
# library's mixed form (PCG dipoles, FP32 FS2 terms, FP64 FS3).
FORMS = {"fp64": ("fp64", {}), "mixed": ("mixed", {})}


def open_context(model, box, device, form):
    from ccpol23_plus_2025_mbmd_b200 import Context
    prec, opts = FORMS[form]
    ctx = Context(model, box.nm, box.box, device=device, precision=prec)
    for k, v in opts.items():
        ctx.set_option(k, v)
    return ctx


def workload_name(nm: int) -> str:
    """The workload both arms time: one hot-path force evaluation of an nm-water box."""
    return (f"{nm} H2O FS2+FS3 hot-path force evaluation (Ewald self/real/recip + "
            "induced-dipole solve + induction forces + FS2 + FS3)")


def ns_per_day(steps_per_s: float) -> float:
    return steps_per_s * DT_PS * 86400.0 / 1000.0


def max_over_ranks(v: float, world: int, device: str = "cuda") -> float:
    """The maximum of v over the ranks (every rank takes part and gets it): per-step times of
    replicas are reported at the slowest rank's pace."""
    if world == 1:
        return v
    import torch
    import torch.distributed as dist
    t = torch.tensor([v], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms while running."""

    def __init__(self, index: int):
        self.index = index
        self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.proc = None

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=self.file, stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        self.file.flush()
        rows = []
        for ln in Path(self.file.name).read_text().splitlines():
            t = [x.strip() for x in ln.split(",")]
            if len(t) >= 9:
                rows.append(t)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        smax = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": max(smax) if smax else None, "reasons": reasons,
                "samples": len(rows)}


def build_inputs(rank: int, config: str = CONFIG):
    from ccpol23_plus_2025_mbmd_b200 import Model, data_dir
    from ccpol23_plus_2025_mbmd_b200.generator import CONFIGS, water_box
    cfg = CONFIGS[config]
    model = Model(data_dir(cfg["variant"]))
    box = water_box(model, cfg["nm"], cfg["box"], cfg["seed"] + rank)
    return model, box, cfg


def time_device(ctx, box, steps, warmup, flush, torch):
    """Device-resident steps: inputs already in HBM, per-step CUDA events on the context's
    (torch's current) stream, L2 flushed between steps outside the events."""
    dev = torch.device("cuda", torch.cuda.current_device())
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    x, y, z, xs, ys, zs = (T(a) for a in (box.x, box.y, box.z, box.xs, box.ys, box.zs))
    f = [torch.zeros_like(xs) for _ in range(3)]
    c2 = [torch.zeros_like(x) for _ in range(3)]
    c3 = [torch.zeros_like(x) for _ in range(3)]
    mu = [torch.zeros_like(xs) for _ in range(3)]
    stream = torch.cuda.current_stream()
    ctx.set_stream(stream.cuda_stream)
    ctx.set_timing(True)
    for _ in range(warmup):
        e = ctx.hot_path_device(x, y, z, xs, ys, zs, box.box, *f, *c2, *c3, *mu)
    torch.cuda.synchronize()
    for t in f:
        t.zero_()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
    phases = []
    launches = 0
    t0 = time.perf_counter()
    for k in range(steps):
        flush.add_(1.0)
        for t in f:  # site forces accumulate (reference semantics): start each step at zero
            t.zero_()
        ev[k][0].record(stream)
        e = ctx.hot_path_device(x, y, z, xs, ys, zs, box.box, *f, *c2, *c3, *mu)
        ev[k][1].record(stream)
        phases.append(ctx.phase_ms())
        launches += ctx.last_launches()
    torch.cuda.synchronize()
    wall = time.perf_counter() - t0
    ms = [a.elapsed_time(b) for a, b in ev]
    forces = np.stack([t.cpu().numpy() for t in f])
    return {"ms": ms, "phases": np.array(phases), "energies": e, "launches": launches,
            "wall_s": wall, "forces": forces,
            "com3": np.stack([t.cpu().numpy() for t in c3]),
            "com2": np.stack([t.cpu().numpy() for t in c2])}


def time_fs3_isolated(ctx, box, torch, reps=5):
    """FS3 kernel time with the three-body terms not overlapped (outside the timed steps):
    the kernel's own speed, for the roofline beside the overlapped figure."""
    dev = torch.device("cuda", torch.cuda.current_device())
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    args = [T(a) for a in (box.x, box.y, box.z, box.xs, box.ys, box.zs)]
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    ctx.set_option("overlap", 0)
    ctx.set_timing(True)
    ms = []
    for k in range(reps + 1):
        ctx.hot_path_device(*args, box.box)
        if k:
            ms.append(ctx.phase_ms()[8])
    ctx.set_option("overlap", 1)
    ctx.set_timing(False)
    return float(np.mean(ms))


def time_e2e(ctx, box, steps, warmup, flush, torch):
    """Through the public host-buffer entry point: H2D of the step's inputs and D2H of its
    forces, COM forces, dipoles and energies inside the timed region."""
    ctx.set_stream(None)
    ctx.set_timing(False)
    for _ in range(warmup):
        ctx.hot_path(box.x, box.y, box.z, box.xs, box.ys, box.zs, box.box)
    torch.cuda.synchronize()
    times = []
    for _ in range(steps):
        flush.add_(1.0)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ctx.hot_path(box.x, box.y, box.z, box.xs, box.ys, box.zs, box.box)
        times.append(time.perf_counter() - t0)
    nm, ld = box.xs.shape
    ns = ctx.model.ns
    npol = ctx.model.npol
    h2d = 8 * (3 * nm + 3 * nm * ld)
    d2h = 8 * (3 * nm * ns + 6 * nm + 3 * nm * npol) + 8 * 16 + 4 * 5
    return times, h2d, d2h


def time_md_steps(model, box, state, prec, steps, device, torch):
    """Whole rigid-water NVE MD steps (2-body term + hot path + nve_1 integrator, state on
    the device, per-step scalars back to the host) from `state`, wall-clock timed around
    ccp_md_nve so that every host round trip of a step is inside."""
    with open_context(model, box, device, prec) as ctx:
        ctx.md_set_state(box.box, state["x"], state["y"], state["z"], state["v"], state["q"],
                         state["j"])
        ctx.md_nve(5, DT_PS)  # warm-up: list sizes, graphs
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        st = ctx.md_nve(steps, DT_PS)
        wall = time.perf_counter() - t0
    return {"ms_per_md_step": wall / steps * 1e3, "ns_day": ns_per_day(steps / wall),
            "steps": steps, "ind_iters_mean": float(np.mean([s["ind_iters"] for s in st]))}


def cpu_baseline(box, cfg, max_seconds=60.0):
    """The oracle's hot path on all host cores for one full step of the same box."""
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle as O
    from ccpol23_plus_2025_mbmd_b200 import data_dir
    O.build()
    cores = os.cpu_count() or 1
    O.set_threads(cores)
    M = O.make_model(O.read_inputs(data_dir(cfg["variant"])), box.nm, box.box)
    t0 = time.perf_counter()
    e, st = O.hot_path(M, box.x, box.y, box.z, box.xs, box.ys, box.zs, box.box)
    dt = time.perf_counter() - t0
    return dt, cores, e, st


def _generator_module():
    """The box generator, loaded from its file without importing the package (whose
    __init__ loads the library): the reference arm must run the oracle alone."""
    import importlib.util
    spec = importlib.util.spec_from_file_location(
        "_ccp_box_generator", ROOT / "ccpol23_plus_2025_mbmd_b200" / "generator.py")
    if spec.name in sys.modules:
        return sys.modules[spec.name]
    mod = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = mod  # its dataclass resolves annotations through sys.modules
    spec.loader.exec_module(mod)
    return mod


def reference_inputs(config=CONFIG, rank=0):
    """The benchmark box built by the oracle alone (its input readers, principal frame and
    site placement; the same seeded generator): bit-identical to build_inputs', with nothing
    of the package imported or loaded.  Returns (oracle module, oracle model, box, config)."""
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle as O
    gen = _generator_module()
    cfg = gen.CONFIGS[config]
    inp = O.read_inputs(ROOT / "ccpol23_plus_2025_mbmd_b200" / "data" / cfg["variant"])
    box = gen.water_box(O.SiteFrame(inp), cfg["nm"], cfg["box"], cfg["seed"] + rank)
    O.build()
    M = O.make_model(inp, box.nm, box.box)
    return O, M, box, cfg


def run_reference(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return
    O, M, box, cfg = reference_inputs()
    cores = os.cpu_count() or 1
    O.set_threads(cores)
    # no warm-up steps: a CPU step has nothing to warm and each one takes seconds
    times = []
    budget = 240.0
    t_start = time.perf_counter()
    for k in range(args.steps):
        t0 = time.perf_counter()
        O.hot_path(M, box.x, box.y, box.z, box.xs, box.ys, box.zs, box.box)
        times.append(time.perf_counter() - t0)
        if time.perf_counter() - t_start > budget:
            break
    s = float(np.mean(times))
    val = ns_per_day(1.0 / s)
    line = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": "ns/day",
        "n_gpus": world, "steps": len(times), "warmup": 0, "ms_per_step": s * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded jittered-lattice water box)",
        "config": {"workload": workload_name(box.nm), "nm": box.nm, "box_A": box.box,
                   "variant": cfg["variant"], "seed": cfg["seed"], "parallelism": "replicas x1"},
        "cpu_baseline": {"value": val, "unit": "ns/day", "cores": cores, "kind": "port",
                         "sample": f"{len(times)} of {args.steps} requested full hot-path "
                                   f"evaluations of the 512-water box (time-capped at "
                                   f"{budget:.0f} s); oracle built with {O.BUILD_FLAGS}, "
                                   f"{cores} OpenMP threads"},
        "e2e": {"value": val, "unit": "ns/day", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_single(which, host_loop=False, config=CONFIG, opts=()):
    import torch
    from ccpol23_plus_2025_mbmd_b200 import Context
    model, box, cfg = build_inputs(0, config)
    dev = torch.device("cuda", 0)
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    args = [T(a) for a in (box.x, box.y, box.z, box.xs, box.ys, box.zs)]
    for prec in (("fp64", "mixed") if which == "both" else (which,)):
        with Context(model, box.nm, box.box, device=0, precision=prec) as ctx:
            ctx.set_timing(True)
            if host_loop:
                ctx.set_option("graph_loop", 0)
            for k, v in opts:
                ctx.set_option(k, v)
            f = [torch.zeros_like(args[3]) for _ in range(3)]
            for _ in range(3):  # the first call sizes lists and builds the dipole-loop graph
                e = ctx.hot_path_device(*args, box.box, *f)
            torch.cuda.synchronize()
            print(json.dumps({"form": prec, "phase_ms": [round(v, 4) for v in ctx.phase_ms()],
                              "launches": ctx.last_launches(), "ind_iters": e["ind_iters"],
                              "n_fs3_triples": e["n_fs3_triples"], "n_fs3_blend": e["n_fs3_blend"],
                              "n_fs2_triples": e["n_fs2_triples"]}), flush=True)


def run_floor(config, steps, warmup, opts=()):
    """The critical-path floor of the evaluation, per form (one JSON line each): the
    Ewald/induction chain alone (self, real, reciprocal, induction), its dipole loop within
    that, the three-body terms alone, FS3 alone, the whole step with the terms overlapping
    (with the loop's and FS3's own durations there) and with them in order on one stream.
    CUDA events on torch's current stream around each evaluation, L2 flushed before each,
    means over `steps` evaluations after `warmup`.  `opts` are (name, value) context options
    set on both forms."""
    import torch
    from ccpol23_plus_2025_mbmd_b200 import _lib
    model, box, cfg = build_inputs(0, config)
    dev = torch.device("cuda", 0)
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    args = [T(a) for a in (box.x, box.y, box.z, box.xs, box.ys, box.zs)]
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=dev)
    chain = _lib.TERM_SELF | _lib.TERM_RSPACE | _lib.TERM_KSPACE | _lib.TERM_INDUCTION
    three = _lib.TERM_FS2 | _lib.TERM_FS3

    def timed(ctx, terms):
        ms, ph = [], []
        for it in range(warmup + steps):
            flush.add_(1.0)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record()
            ctx.terms_device(terms, *args, box.box)
            e1.record()
            torch.cuda.synchronize()
            if it >= warmup:
                ms.append(e0.elapsed_time(e1))
                ph.append(ctx.phase_ms())
        return float(np.mean(ms)), np.mean(ph, axis=0)

    for form in ("fp64", "mixed"):
        with open_context(model, box, 0, form) as ctx:
            ctx.set_stream(torch.cuda.current_stream().cuda_stream)
            ctx.set_timing(True)
            for k, v in opts:
                ctx.set_option(k, v)
            r = {"box": config, "nm": box.nm, "form": form, "options": dict(opts)}
            r["chain_alone_ms"], ph = timed(ctx, chain)
            r["loop_alone_ms"] = float(ph[4])
            r["three_body_alone_ms"], _ = timed(ctx, three)
            r["fs3_alone_ms"], _ = timed(ctx, _lib.TERM_FS3)
            r["step_overlapped_ms"], ph = timed(ctx, _lib.TERM_HOT)
            r["loop_overlapped_ms"], r["fs3_overlapped_ms"] = float(ph[4]), float(ph[8])
            ctx.set_option("overlap", 0)
            r["step_serial_ms"], _ = timed(ctx, _lib.TERM_HOT)
            print(json.dumps({k: round(v, 4) if isinstance(v, float) else v
                              for k, v in r.items()}), flush=True)


def equilibrate(ctx, box, nsteps, temp=298.0, every=20):
    """Velocity-rescaled MD from the synthetic start (its jittered lattice is far from
    equilibrium): every `every` steps the COM velocities and angular momenta are scaled to
    the target temperature.  Returns the state."""
    ctx.md_set_state(box.box, box.x, box.y, box.z, box.v, box.q, box.jb)
    for _ in range(max(nsteps // every, 0)):
        st = ctx.md_nve(every, DT_PS)
        f = np.sqrt(temp / st[-1]["sys_temp"])
        s = ctx.md_get_state()
        ctx.md_set_state(box.box, s["x"], s["y"], s["z"], s["v"] * f, s["q"], s["j"] * f)
    return ctx.md_get_state()


def run_batch(nframes, steps, warmup):
    """Batches of independent 256-water FS3 frames (L = 19.71 A, seed 4004 + f), the
    three-body plus induction terms that the autograd binding evaluates: device-resident
    inputs, frames one by one on one context against one ccp_batch_terms_device call per
    batch (slots 1 / 8 / nframes), with FS3 fused over the frames (one launch set) and not.  Wall time per batch on the host, device synchronised on
    both sides; prints one JSON line, not the headline metric."""
    import torch
    from ccpol23_plus_2025_mbmd_b200 import Batch, Context, Model, data_dir, _lib
    from ccpol23_plus_2025_mbmd_b200.generator import CONFIGS, water_box
    cfg = CONFIGS["c4_256"]
    model = Model(data_dir(cfg["variant"]))
    boxes = [water_box(model, cfg["nm"], cfg["box"], cfg["seed"] + f) for f in range(nframes)]
    dev = torch.device("cuda", 0)
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    x, y, z, xs, ys, zs = (T(np.stack([getattr(b, k) for b in boxes]))
                           for k in ("x", "y", "z", "xs", "ys", "zs"))
    f = [torch.zeros_like(xs) for _ in range(3)]
    terms = _lib.TERM_INDUCTION | _lib.TERM_FS2 | _lib.TERM_FS3
    nm, L = cfg["nm"], cfg["box"]

    def timed(run):
        for _ in range(warmup):
            run()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(steps):
            run()
        torch.cuda.synchronize()
        return (time.perf_counter() - t0) / steps

    out = {}
    with Context(model, nm, L) as c:
        def one_by_one():
            for k in range(nframes):
                c.terms_device(terms, x[k], y[k], z[k], xs[k], ys[k], zs[k], L, f[0][k], f[1][k],
                               f[2][k])
        out["frame_by_frame"] = timed(one_by_one)
    for slots in sorted({1, 8, nframes}):
        for fuse in (1, 0):
            with Batch(model, nm, L, slots=slots) as b:
                b.set_option("fuse_fs3", fuse)
                out[f"batch_slots{slots}_" + ("fs3_fused" if fuse else "fs3_per_frame")] = timed(
                    lambda: b.terms_device(terms, L, x, y, z, xs, ys, zs, *f))
    line = {"metric": f"batch of {nframes} x {nm}-water FS3 frames, three-body + induction",
            "unit": "ms per batch", "steps": steps, "warmup": warmup,
            "config": {"nm": nm, "box_A": L, "variant": cfg["variant"], "seed": cfg["seed"],
                       "frames": nframes},
            **{k: v * 1e3 for k, v in out.items()},
            "frames_per_s": {k: nframes / v for k, v in out.items()}}
    print(json.dumps(line), flush=True)


def run_fort401(steps):
    """The configuration of the only timing the reference ships (its fort.401: 97.59 s for one
    MD step, npt_b ensemble, 256 waters FS2+FS3, 1 MPI rank): a seeded 256-water FS2+FS3 box
    at the C4 density (L = 19.71 A), the device npt_b_1 step (2-body + hot path + integrator)
    timed over `steps` steps after 3 warm-up steps, and the oracle's full force evaluation of
    the same box (2-body + hot path; the integrator is negligible beside it) on 1 host thread
    and on all of them.  Prints one JSON line; not the headline metric."""
    import torch
    from ccpol23_plus_2025_mbmd_b200 import Context, Model, data_dir
    from ccpol23_plus_2025_mbmd_b200.generator import water_box
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle as O
    model = Model(data_dir("fs2fs3"))
    nm, L, seed = 256, 19.71, 4004
    box = water_box(model, nm, L, seed)
    with Context(model, nm, L, device=0) as ctx:
        ctx.md_set_state(L, box.x, box.y, box.z, box.v, box.q, box.jb)
        ctx.md_set_ensemble("npt_b", model.get_double("temp0"), model.get_double("taut"),
                            model.get_double("pres0"), model.get_double("taup"))
        ctx.md_run(3, DT_PS)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ctx.md_run(steps, DT_PS)
        gpu_s = (time.perf_counter() - t0) / steps
    O.build()
    inp = O.read_inputs(data_dir("fs2fs3"))
    pcoord, _, _ = O.principal_frame(inp)
    cpu = {}
    for threads in (1, os.cpu_count() or 1):
        O.set_threads(threads)
        M = O.make_model(inp, nm, L)
        t0 = time.perf_counter()
        O.force_field(M, (True, True), pcoord, box.x, box.y, box.z, box.q, L, box.xs.shape[1])
        cpu[threads] = time.perf_counter() - t0
    line = {"metric": "s per MD step, 256 H2O FS2+FS3, npt_b (the reference's fort.401 case)",
            "reference_published_s_per_step": 97.59,
            "reference_published_note": "fort.401 of the reference: 1 MPI rank on its authors' "
                                        "cluster CPU (hardware unknown)",
            "gpu_s_per_step": gpu_s, "gpu_steps": steps,
            "oracle_force_evaluation_s": {f"{k}_threads": v for k, v in cpu.items()},
            "gpu_speedup_vs_published": 97.59 / gpu_s,
            "gpu_speedup_vs_oracle_1_thread": cpu[1] / gpu_s,
            "config": {"nm": nm, "box_A": L, "variant": "fs2fs3", "seed": seed,
                       "ensemble": "npt_b", "wall_clock_timed": True}}
    print(json.dumps(line), flush=True)


def run_nve(nsteps, nequil):
    """Rigid-water NVE MD on the device (2-body + hot path + nve_1), FP64 and mixed forms from
    the same equilibrated state: time per MD step and the energy drift (linear fit of the
    total energy, kcal/mol per ns).  Prints one JSON line; not the headline metric."""
    import torch
    from ccpol23_plus_2025_mbmd_b200 import Context
    model, box, cfg = build_inputs(0)
    with Context(model, box.nm, box.box, device=0) as ctx:
        s0 = equilibrate(ctx, box, nequil)
    out = {}
    for prec in ("fp64", "mixed"):
        with Context(model, box.nm, box.box, device=0, precision=prec) as ctx:
            ctx.md_set_state(box.box, s0["x"], s0["y"], s0["z"], s0["v"], s0["q"], s0["j"])
            ctx.md_nve(5, DT_PS)  # warm-up: list sizes, graphs
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            st = ctx.md_nve(nsteps, DT_PS)
            wall = time.perf_counter() - t0
        te = np.array([s["te"] for s in st])
        t_ns = np.arange(1, nsteps + 1) * DT_PS * 1e-3
        slope = float(np.polyfit(t_ns, te, 1)[0]) if nsteps > 1 else 0.0
        out[prec] = {"ms_per_md_step": wall / nsteps * 1e3,
                     "ns_day": ns_per_day(nsteps / wall),
                     "drift_kcal_mol_per_ns": slope,
                     "drift_per_molecule_kcal_mol_per_ns": slope / box.nm,
                     "te_first": float(te[0]), "te_last": float(te[-1]),
                     "te_rms_fluct": float(np.std(te)),
                     "temp_mean_K": float(np.mean([s["sys_temp"] for s in st]))}
    line = {"metric": "NVE MD, 512 H2O FS2+FS3 (2-body + hot path + nve_1 integrator)",
            "steps": nsteps, "dt_ps": DT_PS, "wall_clock_timed": True,
            "equilibration": f"{nequil} steps, velocities rescaled to 298 K every 20 steps, FP64",
            "config": {"nm": box.nm, "box_A": box.box, "variant": cfg["variant"], "seed": cfg["seed"]},
            "fp64": out["fp64"], "mixed": out["mixed"],
            "drift_ratio_mixed_over_fp64": (abs(out["mixed"]["drift_kcal_mol_per_ns"]) /
                                             max(abs(out["fp64"]["drift_kcal_mol_per_ns"]), 1e-30))}
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--config", default=CONFIG, choices=[CONFIG, "c5_2048"],
                    help="c5_2048: the same measurement on the 2048-water box (L = 39.40 A)")
    ap.add_argument("--md-steps", type=int, default=100,
                    help="whole NVE MD steps timed per form for the md_step keys (0: skip)")
    ap.add_argument("--md-equil", type=int, default=200,
                    help="velocity-rescaled FP64 steps before the md_step timing")
    ap.add_argument("--single", choices=["fp64", "mixed", "both"],
                    help="three device-resident evaluations per form, phase times of the last "
                         "(profiling; no timing loop)")
    ap.add_argument("--nve", type=int, default=0, metavar="STEPS",
                    help="run STEPS NVE MD steps per form and print the drift line instead")
    ap.add_argument("--nve-equil", type=int, default=4000, metavar="STEPS",
                    help="velocity-rescaled equilibration steps before the NVE run")
    ap.add_argument("--batch", type=int, default=0, metavar="FRAMES",
                    help="time FRAMES 256-water FS3 frames (three-body + induction terms) one "
                         "by one and as one batch call, and print that line instead")
    ap.add_argument("--fort401", action="store_true",
                    help="time the reference's own published case (256 waters, npt_b, one MD "
                         "step) on the device and on 1 and all host threads, and print that line")
    ap.add_argument("--floor", action="store_true",
                    help="print the critical-path floor table (chain, dipole loop, three-body "
                         "terms and FS3 alone, overlapped and in order) per form instead")
    ap.add_argument("--opt", action="append", default=[], metavar="NAME=VALUE",
                    help="with --floor or --single: a context option set on every form (repeatable)")
    ap.add_argument("--host-loop", action="store_true",
                    help="with --single: drive the dipole iteration from the host, so that "
                         "profilers see its kernels")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
        return
    opts = [(kv.split("=", 1)[0], int(kv.split("=", 1)[1])) for kv in args.opt]
    if args.single:
        run_single(args.single, args.host_loop, args.config, opts)
        return
    if args.floor:
        run_floor(args.config, args.steps, args.warmup, opts)
        return
    if args.nve:
        run_nve(args.nve, args.nve_equil)
        return
    if args.batch:
        run_batch(args.batch, args.steps, args.warmup)
        return
    if args.fort401:
        run_fort401(args.steps)
        return
    import torch
    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    from ccpol23_plus_2025_mbmd_b200 import Context
    from ccpol23_plus_2025_mbmd_b200.api import fma_peak_tflops, mufu_peak_tops

    model, box, cfg = build_inputs(rank, args.config)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device="cuda")  # 256 MB > L2
    forms = ["fp64", "mixed"]
    results = {}
    with ClockSampler(local) as clk:
        for prec in forms:
            with open_context(model, box, local, prec) as ctx:
                if world > 1:
                    dist.barrier()
                torch.cuda.synchronize()
                r = time_device(ctx, box, args.steps, args.warmup, flush, torch)
                torch.cuda.synchronize()
                if world > 1:
                    dist.barrier()
                t, h2d, d2h = time_e2e(ctx, box, args.steps, args.warmup, flush, torch)
                r["e2e_s"] = t
                r["h2d"], r["d2h"] = h2d, d2h
                r["fs3_isolated_ms"] = time_fs3_isolated(ctx, box, torch)
                r["fs3_pairs"] = ctx.get_option("fs3_pair_form_active")
                results[prec] = r
        # whole MD steps of both forms from one short velocity-rescaled equilibration
        md = {}
        if args.md_steps > 0:
            with Context(model, box.nm, box.box, device=local, precision="fp64") as ctx:
                s0 = equilibrate(ctx, box, args.md_equil)
            for prec in forms:
                md[prec] = time_md_steps(model, box, s0, prec, args.md_steps, local, torch)
    clocks = clk.summary()
    peak64 = fma_peak_tflops(local, "fp64")
    peak32 = fma_peak_tflops(local, "mixed")
    peak_mufu = mufu_peak_tops(local)

    def agg(v):
        return max_over_ranks(v, world)

    out = {}
    for prec, r in results.items():
        ms = agg(float(np.mean(r["ms"])))
        e2e = agg(float(np.mean(r["e2e_s"])))
        e = r["energies"]
        out[prec] = {"ms_per_step": ms, "ns_day": world * ns_per_day(1e3 / ms),
                     "e2e_ns_day": world * ns_per_day(1.0 / e2e), "e2e_ms": e2e * 1e3,
                     "triples_per_s": world * e["n_fs3_triples"] / (ms * 1e-3),
                     "fs3_ms": float(np.mean(r["phases"][:, 8])),
                     "fs3_isolated_ms": r["fs3_isolated_ms"],
                     "phase_ms": [float(v) for v in r["phases"].mean(0)],
                     "ind_iters": e["ind_iters"], "n_fs3_triples": e["n_fs3_triples"],
                     "n_fs3_blend": e["n_fs3_blend"], "n_fs2_triples": e["n_fs2_triples"],
                     "launches_per_step": r["launches"] / args.steps}
    # each other form against the FP64 form on the same box

    def mol_force_torque(r):
        F = r["forces"]  # (3, nm, ld) site forces of the last step
        tot = F.sum(2) + r["com2"] + r["com3"]
        sx, sy, sz = box.xs, box.ys, box.zs
        tq = np.stack([(sy * F[2] - sz * F[1]).sum(1), (sz * F[0] - sx * F[2]).sum(1),
                       (sx * F[1] - sy * F[0]).sum(1)])
        return tot, tq

    rl = lambda a, b: float(np.linalg.norm(a - b) / np.linalg.norm(b))
    f64 = results["fp64"]
    T64, Q64 = mol_force_torque(f64)
    errs = {}
    for form in forms[1:]:
        fmx = results[form]
        Tmx, Qmx = mol_force_torque(fmx)
        e64, emx = f64["energies"], fmx["energies"]
        er = {"rel_site_force_err": rl(fmx["forces"], f64["forces"]),
              "rel_molecule_force_err": rl(Tmx, T64), "rel_molecule_torque_err": rl(Qmx, Q64),
              "rel_fs3_com_force_err": rl(fmx["com3"], f64["com3"]),
              "rel_fs2_com_force_err": rl(fmx["com2"], f64["com2"])}
        for k in ("fs3pe", "fs2pe", "indpe"):
            er[f"rel_{k}_err"] = abs(emx[k] - e64[k]) / max(abs(e64[k]), 1e-300)
        er["within_1e-5"] = max(er["rel_site_force_err"], er["rel_molecule_force_err"],
                                er["rel_molecule_torque_err"]) <= 1e-5
        errs[form] = er
    # the headline form: the fastest end to end (the reference-facing figure) of the forms
    # that meet the accuracy bar
    ok = ["fp64"] + [f for f in forms[1:] if errs[f]["within_1e-5"]]
    head = max(ok, key=lambda f: out[f]["e2e_ns_day"])
    H = out[head]
    # roofline of the dominant kernel (FS3) of the headline form
    e = results[head]["energies"]
    sums = e["n_fs3_triples"] + e["n_fs3_blend"]
    site_triples = sums * 17 ** 3
    fs3_s, iso_s = H["fs3_ms"] * 1e-3, results[head]["fs3_isolated_ms"] * 1e-3
    ref_flop = FS3_FLOP_PER_SITE_TRIPLE * site_triples
    # by triples (pair form off) the kernel does the reference's work, site triple by site triple
    pairs = results[head]["fs3_pairs"]
    flop = FS3_FLOP_PER_SUM * sums if pairs else ref_flop
    achieved, iso = flop / fs3_s / 1e12, flop / iso_s / 1e12
    peak = peak64  # FS3 is FP64 in both forms
    line = {
        "metric": METRIC if args.config == CONFIG else METRIC_C5,
        "value": out[head]["ns_day"], "unit": "ns/day", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": H["ms_per_step"],
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if head == "fp64" else "f32+f64",
        "data": "synthetic (seeded jittered-lattice water box, 298 K)",
        "config": {"workload": workload_name(box.nm), "nm": box.nm, "box_A": box.box, "variant": cfg["variant"], "seed": cfg["seed"],
                   "form": head, "l2": "flushed between timed steps (256 MB write)",
                   "parallelism": f"replicas x{world}"},
        "triples_per_s": H["triples_per_s"],
        **{f: out[f] for f in forms},
        "mixed_speedup_over_fp64": {
            "device": out["fp64"]["ms_per_step"] / out["mixed"]["ms_per_step"],
            "e2e": out["fp64"]["e2e_ms"] / out["mixed"]["e2e_ms"],
            "fs3_isolated": out["fp64"]["fs3_isolated_ms"] / out["mixed"]["fs3_isolated_ms"]},
        "md_step": ({**md, "workload": f"NVE MD step, {box.nm} H2O FS2+FS3: 2-body + hot path + "
                                       "nve_1 integrator, per-step scalars to the host",
                     "equilibration": f"{args.md_equil} FP64 steps, velocities rescaled to "
                                      "298 K every 20 steps",
                     "timing": "wall clock around ccp_md_nve (host round trips inside)",
                     "mixed_speedup_over_fp64": md["fp64"]["ms_per_md_step"] /
                                                md["mixed"]["ms_per_md_step"]}
                    if md else None),
        **{f"{f}_vs_fp64": errs[f] for f in forms[1:]},
        "e2e": {"value": H["e2e_ns_day"], "unit": "ns/day",
                "h2d_bytes_per_step": results[head]["h2d"], "d2h_bytes_per_step": results[head]["d2h"]},
        "roofline": {"bound": "fp64_pipe",
                     "kernel": "k_fs3_pair<false> + k_fs3_energy" if pairs else "k_fs3",
                     "achieved": achieved, "peak": peak, "unit": "TFLOP/s", "frac": achieved / peak,
                     "peak_source": "measured in this run by an FMA-chain microbenchmark "
                                    "(MEASURED_PEAKS.json has no FP32/FP64 figure)",
                     "work": (f"{FS3_FLOP_PER_SUM:.0f} flop per sum (three visits of the pair "
                              f"kernel and one energy sum) x {sums} sums per evaluation, as the "
                              "kernels execute them" if pairs else
                              f"{FS3_FLOP_PER_SITE_TRIPLE:.0f} flop per site triple x "
                              f"{site_triples} site triples"),
                     "duration_ms": H["fs3_ms"],
                     "note": "achieved uses the kernels' duration in the timed steps, where they "
                             "share the GPU with the Ewald/induction kernels; 'isolated' is the "
                             "same with the three-body terms not overlapped",
                     "isolated": {"duration_ms": iso_s * 1e3, "achieved": iso,
                                  "frac": iso / peak},
                     # the reference's work for the same sums, which the kernels regroup into
                     # less: a rate of results, not of the pipe
                     "reference_work": {"flop_per_site_triple": FS3_FLOP_PER_SITE_TRIPLE,
                                        "site_triples": site_triples,
                                        "tflop_per_s": ref_flop / fs3_s / 1e12,
                                        "tflop_per_s_isolated": ref_flop / iso_s / 1e12},
                     # DRAM bytes (read + write) of the pair and the energy kernel (377 and 85
                     # MB) from an ncu capture at 512 waters (31417 triples): the pairs' tables,
                     # 170 MB there, which L2 does not hold; on another box scaled by its triple
                     # count
                     "traffic": 4.62e8 * e["n_fs3_triples"] / 31417.0,
                     "traffic_unit": "bytes per launch"
                                     + ("" if args.config == CONFIG else
                                        " (ncu capture at 512 waters scaled by the triple count)")},
        "gpu_launches": int(results[head]["launches"]),
        "clocks": clocks,
        "peaks_tflops": {"fp64_fma": peak64, "fp32_fma": peak32, "mufu_exp_tops": peak_mufu},
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline and args.config == CONFIG:
        dt, cores, eo, st = cpu_baseline(box, cfg)
        line["cpu_baseline"] = {"value": ns_per_day(1.0 / dt), "unit": "ns/day", "cores": cores,
                                "kind": "port",
                                "sample": f"1 full hot-path evaluation of the same {box.nm}-water box "
                                          f"({dt:.1f} s on {cores} threads; oracle built with "
                                          "gcc -O3 -fopenmp -ffp-contract=off)"}
        Fo = np.stack([st.fxs, st.fys, st.fzs])
        line["parity_vs_oracle"] = {
            f"{f}_rel_force_err": float(np.linalg.norm(results[f]["forces"] - Fo) /
                                        np.linalg.norm(Fo)) for f in forms}
    if world > 1:
        torch.cuda.synchronize()
        dist.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)


if __name__ == "__main__":
    main()
