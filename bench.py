#!/usr/bin/env python
"""Benchmark: gridded samples/s of batched 2-D radial adjoint reconstruction.

Workload (the batched dynamic 2-D radial configuration): 96 frames x 34
golden-angle spokes x 384 readout samples, 32 coils, complex64, moving-ellipse
phantom (analytic k-space, linear-phase coil maps, 30 dB noise); Kaiser-Bessel
width 4 on a sigma = 2 grid (384^2) for a 192^2 image, analytic ramp (Ram-Lak)
DCF, deapodised, cropped and combined by root sum of squares.  One step = one
call reconstructing all 96 frames x 32 coils (40 108 032 gridded samples).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

`value`: device-resident inputs (321 MB of samples, larger than the 129 MB L2,
so no flush is needed between steps).  `e2e`: the same reconstruction through
the host-buffer entry point, with the samples and trajectory copied from
pinned host memory and the images copied back inside every step (the copies
overlap the frame passes); the median of five timed windows of the same
steps, every window listed.  `--impl reference` times the reference's CPU path
(radial_linear_gridding2_adjoint + ramp DCF, the C restatement that is
bit-identical to it) on a bounded sample of the same workload over all host
cores.  Under torchrun every rank reconstructs its own batch (replicas, weak
scaling, no collective on the data path).
"""
from __future__ import annotations

import argparse
import ctypes
import json
import math
import os
import re
import statistics
import subprocess
import sys
import threading
import time
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

FRAMES, SPOKES, READOUT, COILS = 96, 34, 384, 32
E2E_WINDOWS = 5  # timed windows of the end-to-end measurement (median reported)
IMAGE, GRID, WIDTH = 192, 384, 4
METRIC = "gridded samples/s"
WORKLOAD = "batched dynamic 2D radial adjoint (KB W=4, sigma=2) + RSS"


def workload_config(extra: dict | None = None) -> dict:
    cfg = {"workload": WORKLOAD, "frames": FRAMES, "spokes_per_frame": SPOKES, "readout": READOUT, "coils": COILS,
           "image": IMAGE, "grid": GRID, "kernel": "kaiser_bessel", "kernel_width": WIDTH, "oversampling": 2.0,
           "dcf": "analytic ramp (Ram-Lak)", "output": f"rss float32 [{FRAMES},{IMAGE},{IMAGE}]",
           "l2": f"inputs larger than L2 ({FRAMES * SPOKES * READOUT * COILS * 8 / 1e6:.0f} MB samples)"}
    if extra:
        cfg.update(extra)
    return cfg


def make_inputs(seed: int = 7):
    from kspacejet_gb300 import synth

    traj, ksp = synth.dynamic_radial(FRAMES, SPOKES, READOUT, COILS, seed=seed, image=IMAGE, snr_db=30.0)
    return np.ascontiguousarray(traj, dtype=np.float32), np.ascontiguousarray(ksp, dtype=np.complex64)


# --------------------------------------------------------------- clocks

class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    """nvidia-smi sampled every 25 ms from before the first timed region to after
    the last; summary() keeps the samples that arrived inside the timed windows
    (host monotonic clock, 60 ms of slack for the tool's reporting delay)."""

    def __init__(self, device_index: int):
        self.device_index = device_index
        self.proc = None
        self.lines: list[tuple[float, str]] = []
        self.windows: list[tuple[float, float]] = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.device_index}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "25"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except (OSError, FileNotFoundError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append((time.monotonic(), line.strip()))

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def window(self):
        """Context manager marking one timed region."""
        sampler = self

        class _W:
            def __enter__(self):
                self.t0 = time.monotonic()

            def __exit__(self, *a):
                sampler.windows.append((self.t0, time.monotonic()))
        return _W()

    def summary(self) -> dict:
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        inside = [ln for t, ln in self.lines if any(a <= t <= b + 0.06 for a, b in self.windows)]
        for line in inside:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        loaded = [s for s in sm if s > 0.5 * max(sm)] or sm
        return {"sm_mhz": statistics.median(loaded), "sm_max_mhz": max(smax), "reasons": sorted(reasons),
                "samples": len(sm), "timed_windows": len(self.windows)}


# --------------------------------------------------------- CPU baseline

def _single_thread_rate(task, pairs, budget_s: float = 1.5) -> tuple[float, int]:
    """Gridded samples/s of `task` run one (frame, coil) image after another
    on the calling thread for about `budget_s` (at least one image)."""
    done = samples = 0
    t0 = time.perf_counter()
    while done < len(pairs):
        samples += task(pairs[done])
        done += 1
        if time.perf_counter() - t0 >= budget_s:
            break
    return samples / (time.perf_counter() - t0), done


def cpu_reference_rate(traj: np.ndarray, ksp: np.ndarray, budget_s: float = 2.5, min_pairs: int = 0):
    """Gridded samples/s of the reference's CPU path (ramp DCF + linear
    gridding + separable inverse DFT, one (frame, coil) image per task) on all
    host cores.  Uses the compiled reference where it was built on this
    machine, else the C restatement that is bit-identical to it."""
    import oracle

    try:
        impl, kind = oracle.Reference(), "reference"
    except FileNotFoundError:
        impl, kind = oracle.Oracle(), "port"
    cores = os.cpu_count() or 1
    rng = np.random.default_rng(0)
    pairs = [(int(f), int(c)) for f, c in zip(rng.integers(0, FRAMES, 4096), rng.integers(0, COILS, 4096))]
    dcfs = {}

    def task(fc):
        f, c = fc
        d = dcfs.get(f)
        if d is None:
            d = impl.ramp_dcf(traj[f])
            dcfs[f] = d
        impl.linear_gridding(IMAGE, IMAGE, ksp[f, c], traj[f], d)
        return traj.shape[1]

    done = 0
    samples = 0
    t0 = time.perf_counter()
    with ThreadPoolExecutor(max_workers=cores) as pool:
        while True:
            batch = pairs[done:done + cores]
            samples += sum(pool.map(task, batch))
            done += len(batch)
            el = time.perf_counter() - t0
            if (el >= budget_s and done >= min_pairs) or done >= len(pairs):
                break
    el = time.perf_counter() - t0
    single, single_n = _single_thread_rate(task, pairs[done:] or pairs)
    return {"value": samples / el, "unit": METRIC, "cores": cores, "kind": kind,
            "single_thread_value": single, "single_thread_images": single_n,
            "sample": f"{done} (frame, coil) images of the workload ({traj.shape[1]} samples each) through "
                      f"radial_linear_gridding2_adjoint with ramp DCF on a {IMAGE}x{IMAGE} grid (the reference's "
                      f"direct-DFT fallback for a non-power-of-two axis), {cores} threads, {el:.2f} s wall"}


def cpu_kb_rate(traj: np.ndarray, ksp: np.ndarray, budget_s: float = 3.0, width: int = WIDTH):
    """Gridded samples/s of the same Kaiser-Bessel reconstruction as a
    single-precision CPU program (the oracle's restatement with an FFT: float
    gridding, mixed-radix FFT of the grid rows and of the kept columns, crop,
    deapodisation), one (frame, coil) image per task on all host cores.  The
    reference has no Kaiser-Bessel path, so this is a restatement, not the
    reference."""
    import oracle

    impl = oracle.Oracle()
    cores = os.cpu_count() or 1
    rng = np.random.default_rng(1)
    pairs = [(int(f), int(c)) for f, c in zip(rng.integers(0, FRAMES, 4096), rng.integers(0, COILS, 4096))]
    dcfs = {}

    def task(fc):
        f, c = fc
        d = dcfs.get(f)
        if d is None:
            d = np.hypot(traj[f, :, 0], traj[f, :, 1]).astype(np.float32)
            dcfs[f] = d
        impl.kb_gridding_f32(GRID, IMAGE, ksp[f, c], traj[f], d, width=width)
        return traj.shape[1]

    done = samples = 0
    t0 = time.perf_counter()
    with ThreadPoolExecutor(max_workers=cores) as pool:
        while True:
            batch = pairs[done:done + cores]
            samples += sum(pool.map(task, batch))
            done += len(batch)
            el = time.perf_counter() - t0
            if el >= budget_s or done >= len(pairs):
                break
    el = time.perf_counter() - t0
    single, single_n = _single_thread_rate(task, pairs[done:] or pairs)
    return {"value": samples / el, "unit": METRIC, "cores": cores, "kind": "port",
            "single_thread_value": single, "single_thread_images": single_n,
            "sample": f"restatement, not reference (the reference has no Kaiser-Bessel path): {done} (frame, coil) "
                      f"images of the workload ({traj.shape[1]} samples each), KB W={width} gridding on the "
                      f"{GRID}^2 grid, FFT of every grid row and of the {IMAGE} kept columns, crop and "
                      f"deapodisation in float32, {cores} threads, {el:.2f} s wall"}


def accuracy_check(rss: np.ndarray, traj: np.ndarray, ksp: np.ndarray, frames, width: int = WIDTH,
                   pixels: int = 256) -> dict:
    """Relative L2 error of RSS images the timed call wrote, against (a) the
    RSS of the FP64 restatement of the same Kaiser-Bessel algorithm over every
    coil and (b) the RSS of the exact FP64 direct NUDFT of the DCF-weighted
    samples at `pixels` seeded pixels.  Outside every timed region."""
    import oracle

    orc = oracle.Oracle()
    cores = os.cpu_count() or 1
    rng = np.random.default_rng(17)
    flat = rng.choice(IMAGE * IMAGE, size=pixels, replace=False)
    pix = np.stack([flat // IMAGE, flat % IMAGE], axis=-1)
    o = (IMAGE - 1) / 2.0
    worst_same = worst_exact = 0.0
    with ThreadPoolExecutor(max_workers=cores) as pool:
        for f in frames:
            t64 = traj[f].astype(np.float64)
            d64 = np.hypot(t64[:, 0], t64[:, 1])
            coils = list(pool.map(lambda c: orc.kb_gridding(GRID, IMAGE, ksp[f, c].astype(np.complex128), t64, d64,
                                                            width=width), range(ksp.shape[1])))
            ref = np.sqrt(sum(np.abs(x) ** 2 for x in coils))
            exact = list(pool.map(lambda c: orc.direct_adjoint_at(pix, ksp[f, c].astype(np.complex128) * d64, t64, o, o),
                                  range(ksp.shape[1])))
            ref_exact = np.sqrt(sum(np.abs(x) ** 2 for x in exact))
            worst_same = max(worst_same, oracle.rel_l2(rss[f], ref))
            worst_exact = max(worst_exact, oracle.rel_l2(rss[f][pix[:, 0], pix[:, 1]], ref_exact))
    return {"rel_l2_vs_fp64_same_algorithm": worst_same, "rel_l2_vs_exact_nudft": worst_exact,
            "frames_checked": [int(f) for f in frames], "coils": int(ksp.shape[1]), "output": "rss",
            "exact_nudft_pixels": pixels, "kernel_width": width,
            "note": "max over the checked frames; FP64 Kaiser-Bessel restatement over all pixels, exact FP64 "
                    "direct NUDFT of the DCF-weighted samples at seeded pixels"}


def dropin_leg(steps: int, warmup: int) -> dict:
    """The drop-in operator itself: radial_gridding_reconstruct (linear
    gridding, sigma 1, ramp DCF) at the reference envelope's anchor shape
    (256^2 image, 65 536 samples, 8 coils) fired through the GPU plug-in with
    host buffers (every firing copies in, computes and copies out), next to the
    reference's CPU path on the same shape over all host cores."""
    import oracle
    import kspacejet_gb300
    from kspacejet_gb300 import host as H, synth

    n, c = 256, 8
    tr = synth.golden_angle_radial(512, 128)  # 65 536 samples, |k| <= pi
    m = tr.shape[0]
    ks = synth.multicoil_kspace(tr, n, c, seed=5)
    mod = H.ProviderModule(kspacejet_gb300.NONCARTESIAN_PLUGIN)
    try:
        kin, tin = H.aligned_copy(ks), H.aligned_copy(tr.ravel())
        out = H.aligned((n * n * c,), np.complex64)
        with mod.instance("radial_gridding_reconstruct", H.radial_config(c, n, n, m)) as inst:
            def fire():
                r = inst.fire([(kin, H.TYPE_KSPACE, 0), (tin, H.TYPE_TRAJECTORY, 1)], out, H.TYPE_COIL_IMAGE,
                              scratch_bytes=H.radial_scratch_bytes(n, n, m))
                if r.status != 0:
                    raise RuntimeError(f"plug-in firing failed: {r.status} {r.error}")
            for _ in range(max(warmup, 3)):
                fire()
            t0 = time.perf_counter()
            for _ in range(steps):
                fire()
            gpu_s = (time.perf_counter() - t0) / steps
    finally:
        mod.close()
    try:
        impl, kind = oracle.Reference(), "reference"
    except FileNotFoundError:
        impl, kind = oracle.Oracle(), "port"
    cores = os.cpu_count() or 1
    dcf = impl.ramp_dcf(tr)
    reps = max(1, cores // c)
    t0 = time.perf_counter()
    with ThreadPoolExecutor(max_workers=cores) as pool:
        list(pool.map(lambda i: impl.linear_gridding(n, n, ks[i % c], tr, dcf), range(reps * c)))
    cpu_s = (time.perf_counter() - t0) / reps
    return {"operator": "radial_gridding_reconstruct", "shape": {"image": n, "samples": m, "channels": c},
            "path": "GPU plug-in fired through the C-ABI firing host, pageable host payloads, copies inside",
            "gpu_ms_per_firing": gpu_s * 1e3, "gpu_samples_per_s": c * m / gpu_s,
            "cpu_ms_per_frame": cpu_s * 1e3, "cpu_samples_per_s": c * m / cpu_s,
            "cpu": {"kind": kind, "cores": cores, "what": "ramp DCF + radial_linear_gridding2_adjoint per coil, "
                                                           "one coil per thread"},
            "speedup": cpu_s / gpu_s, "timing": "host wall clock per firing (the firing is synchronous)"}


# ------------------------------------------------------------ GPU arm

def dist_setup(n_gpus: int):
    if int(os.environ.get("WORLD_SIZE", "1")) > 1:
        import torch.distributed as dist

        backend = "gloo"
        dist.init_process_group(backend=backend)
        return dist, dist.get_rank(), dist.get_world_size(), int(os.environ.get("LOCAL_RANK", "0"))
    return None, 0, 1, 0


def max_over_ranks(dist, *values: float) -> tuple[float, ...]:
    """The per-rank timings reduced to their maximum over all ranks (the
    slowest replica sets the whole job's time); unchanged on one process."""
    if dist is None:
        return tuple(float(v) for v in values)
    import torch

    t = torch.tensor([float(v) for v in values], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return tuple(float(v) for v in t.tolist())


def read_traffic() -> float | None:
    """dram__bytes_read.sum + dram__bytes_write.sum per launch of the dominant
    kernel from the committed ncu summary (profiles/)."""
    p = ROOT / "profiles" / "k_rows_dynamic2d.md"
    if not p.exists():
        return None
    m = re.search(r"traffic_bytes_per_full_launch:\s*([0-9.eE+]+)", p.read_text())
    return float(m.group(1)) if m else None


def kernel_bytes(g, entries: int) -> dict:
    """Algorithmic HBM bytes per launch of each kernel of one call."""
    F, C, M = g.frames, g.channels, g.samples
    N, G = IMAGE, GRID
    rec = 16 + 8 * WIDTH                      # per-sample record written by k_prepare
    entry = 8 + 4 * WIDTH                     # per list entry as the row pass reads it
    inter = F * C * G * N * 8                 # row-transformed grid, kept columns only
    return {
        "k_rows": F * M * C * 8 + entries * entry + inter,
        "k_cols": inter + F * N * N * 4,
        "k_place": entries * entry + F * M * rec,
        "k_samples_coil_last": 2 * F * C * M * 8,
        "k_prepare": F * M * 8 + F * M * rec,
    }


def width6_leg(g4_tuning_note: str, k, t, traj_h, ksp_h, dev, steps: int, warmup: int) -> dict:
    """The same workload with Kaiser-Bessel width 6: the form whose
    approximation error against the exact NUDFT is below 1e-5 (width 4 is
    ~4e-4).  Device-resident inputs, tuned, CUDA events; accuracy of its
    output on one frame."""
    import torch
    from kspacejet_gb300 import gpu

    g = gpu.kb_gridding(image=IMAGE, grid=GRID, channels=COILS, samples=traj_h.shape[1], frames=FRAMES, width=6,
                        output=gpu.OUTPUT_RSS)
    out = g.new_output(dev)
    ws = g.new_workspace(dev)
    tuning = g.tune(k, t, out, ws)
    for _ in range(warmup):
        g.run(k, t, out, ws, tuning=tuning)
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        g.run(k, t, out, ws, tuning=tuning)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / steps
    acc = accuracy_check(out.cpu().numpy(), traj_h, ksp_h, frames=(FRAMES // 3,), width=6)
    del ws
    return {"kernel_width": 6, "ms_per_step": ms, "value": FRAMES * COILS * traj_h.shape[1] / (ms / 1e3),
            "unit": "samples/s", "accuracy": acc,
            "tuning": {"coil_group": tuning.coil_group, "column_block": tuning.column_block,
                       "frames_per_pass": tuning.frames_per_pass or (FRAMES + 1) // 2,
                       "rows_blocks_per_sm": tuning.rows_blocks_per_sm}}


def run_ours(args) -> dict | None:
    import torch

    from kspacejet_gb300 import gpu

    dist, rank, world, local_rank = dist_setup(args.gpus)
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    traj_h, ksp_h = make_inputs(seed=7 + rank)
    cpu = cpu_kb_rate(traj_h, ksp_h) if rank == 0 else None
    cpu_linear = cpu_reference_rate(traj_h, ksp_h) if rank == 0 else None

    g = gpu.kb_gridding(image=IMAGE, grid=GRID, channels=COILS, samples=traj_h.shape[1], frames=FRAMES, width=WIDTH,
                        output=gpu.OUTPUT_RSS)
    k = torch.from_numpy(ksp_h).to(dev)
    t = torch.from_numpy(traj_h).to(dev)
    out = g.new_output(dev)
    ws = g.new_workspace(dev)
    stream = torch.cuda.current_stream()
    clocks = ClockSampler(local_rank).__enter__()
    if args.tuning:
        # a fixed tuning (coil_group, column_block, frames_per_pass, rows_blocks_per_sm, coil_parts), e.g. to
        # profile the kernels the autotuner picks in a plain run (its candidate timings are not valid under ncu)
        vals = [int(v) for v in args.tuning.split(",")]
        cg, cb, fpp, rb, parts = vals[:5]
        colp = vals[5] if len(vals) > 5 else 0
        tuning = gpu.GriddingTuning(ctypes.sizeof(gpu.GriddingTuning), cg, cb, 0, fpp, rb, parts, colp)
    else:
        tuning = g.tune(k, t, out, ws)
    for _ in range(args.warmup):
        g.run(k, t, out, ws, tuning=tuning)
    torch.cuda.synchronize()
    _, _, entries = None, None, None
    cw, off, smp = g.binning(ws, tuning)
    entries = int(off[-1])

    def barrier():
        if dist is not None:
            dist.barrier()

    # ---- the batched call captured once in a CUDA graph (all kernels, one replay per step)
    graph = None
    try:
        graph = torch.cuda.CUDAGraph()
        side = torch.cuda.Stream()
        side.wait_stream(stream)
        with torch.cuda.stream(side):
            g.run(k, t, out, ws, tuning=tuning)
        stream.wait_stream(side)
        with torch.cuda.graph(graph):
            g.run(k, t, out, ws, tuning=tuning)
        for _ in range(args.warmup):
            graph.replay()
        torch.cuda.synchronize()
    except Exception as exc:  # capture is an optimisation; the direct path stays measured
        graph = None
        graph_error = repr(exc)

    def step():
        if graph is not None:
            graph.replay()
        else:
            g.run(k, t, out, ws, tuning=tuning)

    # ---- value: device-resident inputs
    barrier()
    torch.cuda.synchronize()
    with clocks.window():
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            step()
        e1.record(stream)
        torch.cuda.synchronize()
    barrier()
    ms = e0.elapsed_time(e1) / args.steps
    # launches inside the timed region: a graph replays the captured call's launches
    per_call_launches = None

    # ---- the same call issued directly (launch count; the ncu launch list's range)
    l0 = gpu.launch_count()
    d0 = torch.cuda.Event(enable_timing=True)
    d1 = torch.cuda.Event(enable_timing=True)
    torch.cuda.nvtx.range_push("ksj_timed")  # ncu --nvtx --nvtx-include ksj_timed/ lists exactly these launches
    with clocks.window():
        d0.record(stream)
        for _ in range(args.steps):
            g.run(k, t, out, ws, tuning=tuning)
        d1.record(stream)
        torch.cuda.synchronize()
    torch.cuda.nvtx.range_pop()
    per_call_launches = (gpu.launch_count() - l0) // args.steps
    # ---- per-kernel event timing (roofline): the tuned call with all frames in one
    # pass, so no two of its launches overlap and each launch's events time it alone
    # (the tuned call may run two passes concurrently on two streams)
    tuning_k = gpu.GriddingTuning(ctypes.sizeof(gpu.GriddingTuning), tuning.coil_group, tuning.column_block,
                                  tuning.list_capacity, FRAMES, tuning.rows_blocks_per_sm, tuning.coil_parts,
                                  tuning.column_pass)
    for _ in range(2):
        g.run(k, t, out, ws, tuning=tuning_k)
    torch.cuda.synchronize()
    gpu.timing_reset()
    gpu.timing_enable(True)
    for _ in range(args.steps):
        g.run(k, t, out, ws, tuning=tuning_k)
    torch.cuda.synchronize()
    gpu.timing_enable(False)
    kernels = gpu.timing_read()
    direct_ms = d0.elapsed_time(d1) / args.steps
    launches = per_call_launches * args.steps

    # ---- per-frame loop: the same 96 frames as 96 one-frame calls
    g1 = gpu.kb_gridding(image=IMAGE, grid=GRID, channels=COILS, samples=traj_h.shape[1], frames=1, width=WIDTH,
                         output=gpu.OUTPUT_RSS)
    ws1 = g1.new_workspace(dev)
    out1 = g1.new_output(dev)
    for f in range(3):
        g1.run(k[f:f + 1], t[f:f + 1], out1, ws1)
    torch.cuda.synchronize()
    p0 = torch.cuda.Event(enable_timing=True)
    p1 = torch.cuda.Event(enable_timing=True)
    p0.record(stream)
    for f in range(FRAMES):
        g1.run(k[f:f + 1], t[f:f + 1], out1, ws1)
    p1.record(stream)
    torch.cuda.synchronize()
    per_frame_ms = p0.elapsed_time(p1)

    # ---- e2e: pinned host buffers through the host-buffer entry point
    # (ksj_gpu_gridding_adjoint_host): every step copies the samples and the
    # trajectory in and the images out, overlapped with the passes
    kh = torch.from_numpy(ksp_h).pin_memory()
    th = torch.from_numpy(traj_h).pin_memory()
    oh = torch.empty(out.shape, dtype=out.dtype).pin_memory()
    wsh = g.new_host_workspace(dev)
    for _ in range(2):
        g.run_host(kh, th, oh, wsh, tuning=tuning)
    # E2E_WINDOWS windows of exactly `steps` steps each, every one bracketed
    # by a barrier and a synchronize; the median is reported.  Each step
    # issues ~30 host calls (copies, events, launches), so a host-side stall
    # (about one window in six on the GB300 host measured) drains the GPU queue and
    # adds ~1 ms per step to that window; the median of five is robust to it
    # and every window is listed in the line.
    e2e_windows = []
    for _ in range(E2E_WINDOWS):
        barrier()
        torch.cuda.synchronize()
        x0 = torch.cuda.Event(enable_timing=True)
        x1 = torch.cuda.Event(enable_timing=True)
        with clocks.window():
            x0.record(stream)
            for _ in range(args.steps):
                g.run_host(kh, th, oh, wsh, tuning=tuning)
            x1.record(stream)
            torch.cuda.synchronize()
        e2e_windows.append(x0.elapsed_time(x1) / args.steps)
    clocks.__exit__(None, None, None)
    barrier()
    e2e_ms = statistics.median(e2e_windows)
    if not np.isfinite(oh.numpy()).all():
        raise RuntimeError("non-finite reconstruction")

    # ---- outside every timed region: accuracy of the timed call's output,
    # the width-6 form, and the drop-in operator through its plug-in
    accuracy = width6 = dropin = None
    if rank == 0:
        step()
        torch.cuda.synchronize()
        accuracy = accuracy_check(out.cpu().numpy(), traj_h, ksp_h, frames=(0, FRAMES // 2))
        if not args.skip_extra:
            width6 = width6_leg("", k, t, traj_h, ksp_h, dev, args.steps, args.warmup)
            dropin = dropin_leg(args.steps, args.warmup)
    served = None
    if rank == 0 and not args.skip_extra:
        del ws
        torch.cuda.empty_cache()
        srv = run_serve(args)
        served = {k2: srv[k2] for k2 in ("value", "serial_value", "vs_serial", "p50_ms", "p99_ms", "serial_p50_ms",
                                         "serial_p99_ms", "poisson_rate_per_s")}
        served.update({"unit": "samples/s", "requests": srv["config"]["requests"],
                       "batches": srv["results"]["served"]["burst"]["batches"],
                       "workload": srv["config"]["workload"], "serial": srv["config"]["serial"],
                       "served": srv["config"]["served"],
                       "note": "value = burst throughput of the served loop (median of 3 bursts); p50/p99 under "
                               "Poisson arrivals at 90 % of the serial path's burst throughput"})

    ms, e2e_ms = max_over_ranks(dist, ms, e2e_ms)
    if rank != 0:
        return None

    per_step = FRAMES * COILS * traj_h.shape[1]
    value = world * per_step / (ms / 1000.0)
    e2e = world * per_step / (e2e_ms / 1000.0)

    # roofline of the dominant kernel
    peaks = {}
    pp = ROOT / "MEASURED_PEAKS.json"
    if pp.exists():
        peaks = json.loads(pp.read_text())
    peak = peaks.get("hbm_gbs")
    peak_src = "measured" if peak else "fallback"
    peak = peak or 6800.0
    bytes_per = kernel_bytes(g, entries)
    dom = max(kernels, key=lambda kv: kv[2]) if kernels else None
    roofline = None
    per_kernel = {}
    calls = args.steps  # per-kernel totals come from the direct (event-timed) pass of args.steps calls
    for name, n, tot in kernels:
        avg = tot / max(n, 1)
        if name in bytes_per:
            bytes_per[name] = bytes_per[name] * calls / max(n, 1)  # per launch (a call may launch a kernel per pass)
        entry = {"launches": n, "avg_ms": round(avg, 4), "share": round(tot / max(sum(x[2] for x in kernels), 1e-9), 4)}
        if name in bytes_per:
            entry["algorithmic_GBps"] = round(bytes_per[name] / (avg / 1000.0) / 1e9, 1)
        per_kernel[name] = entry
    if dom is not None:
        name, n, tot = dom
        avg_s = tot / max(n, 1) / 1000.0
        ach = bytes_per.get(name, 0) / avg_s / 1e9
        traffic = read_traffic() if name == "k_rows" else None
        roofline = {"bound": "hbm", "kernel": name, "achieved": round(ach, 1), "peak": peak, "unit": "GB/s",
                    "frac": round(ach / peak, 4), "peak_source": f"{peak_src} hbm_gbs",
                    "algorithmic_bytes_per_launch": bytes_per.get(name), "traffic": traffic,
                    "timing": "CUDA events around each launch of the tuned call run with all frames in one "
                              "pass (no concurrent launches)"}
    return {
        "metric": METRIC, "value": value, "unit": "samples/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32 (complex64 samples, float32 gridding/FFT)", "data": "synthetic",
        "config": workload_config({"parallelism": f"replicas x{world}" if world > 1 else "single GPU",
                                   "tuning": {"coil_group": tuning.coil_group, "column_block": tuning.column_block,
                                              "frames_per_pass": tuning.frames_per_pass or
                                              ((FRAMES + 1) // 2 if FRAMES >= 4 else FRAMES),
                                              "rows_blocks_per_sm": tuning.rows_blocks_per_sm,
                                              "coil_parts": tuning.coil_parts or 1,
                                              "column_pass": "persistent ring" if tuning.column_pass == 2
                                              else "one CTA per column"},
                                   "gridded_samples_per_step_per_gpu": per_step}),
        "e2e": {"value": e2e, "unit": "samples/s", "ms_per_step": e2e_ms,
                "h2d_bytes_per_step": int(ksp_h.nbytes + traj_h.nbytes), "d2h_bytes_per_step": int(out.numel() * 4),
                "windows_ms_per_step": [round(x, 4) for x in e2e_windows],
                "note": f"median of {E2E_WINDOWS} windows of {args.steps} steps each (host-side stalls occasionally "
                        "slow one window)"},
        "gpu_launches": int(launches),
    "batched": {"graph_replay": graph is not None, "ms_per_step_graph_or_direct": ms,
                "ms_per_step_direct": direct_ms, "per_frame_loop_ms_per_step": per_frame_ms,
                "speedup_vs_per_frame_loop": per_frame_ms / ms, "launches_per_call": per_call_launches},
        "roofline": roofline, "kernels": per_kernel,
        "clocks": clocks.summary(),
        "accuracy": accuracy,
        "cpu_baseline": cpu,
        "reference_cpu_linear": cpu_linear,
        "width6": width6,
        "dropin": dropin,
        "serve": served,
    }


def run_reference(args) -> dict | None:
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return None
    traj_h, ksp_h = make_inputs()
    per = []
    cpu = None
    for i in range(args.warmup + args.steps):
        r = cpu_reference_rate(traj_h, ksp_h, budget_s=1.0, min_pairs=os.cpu_count() or 1)
        if i >= args.warmup:
            per.append(r)
            cpu = r
    value = statistics.median(p["value"] for p in per)
    cpu = dict(cpu)
    cpu["value"] = value
    ms = FRAMES * COILS * traj_h.shape[1] / value * 1000.0
    return {"metric": METRIC, "value": value, "unit": "samples/s", "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic", "impl": "reference",
            "config": workload_config({"note": "reference CPU path on a bounded sample of each step's images; "
                                               "ms_per_step extrapolated to the full 96x32-image step"}),
            "e2e": {"value": value, "unit": "samples/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "cpu_baseline": cpu}


# ------------------------------------------------------- served stream

SERVE_READOUTS = (128, 256, 384, 512)


def serve_workload(n: int, seed: int):
    """n slice requests: readout uniform in {128,256,384,512}, spokes uniform in
    64..805, coils uniform in 8..32, image = readout/2 on a readout^2 grid
    (sigma = 2, KB W=4), ramp DCF, RSS output.  Inputs are pinned host memory;
    the k-space of every request is a prefix of one seeded random buffer (the
    inputs are read-only, so requests may share it)."""
    import torch
    from kspacejet_gb300 import serve, synth

    rng = np.random.default_rng(seed)
    shapes = [(int(rng.choice(SERVE_READOUTS)), int(rng.integers(64, 806)), int(rng.integers(8, 33)))
              for _ in range(n)]
    biggest = max(r * sp * c for r, sp, c in shapes)
    base = torch.from_numpy((rng.standard_normal(biggest) + 1j * rng.standard_normal(biggest)).astype(np.complex64))
    base = base.pin_memory()
    trajs = {}
    reqs = []
    for ro, sp, co in shapes:
        if (ro, sp) not in trajs:
            trajs[(ro, sp)] = torch.from_numpy(synth.golden_angle_radial(ro, sp)).pin_memory()
        tr = trajs[(ro, sp)]
        m = ro * sp
        out = torch.empty((ro // 2, ro // 2), dtype=torch.float32).pin_memory()
        r = serve.Request(image=ro // 2, grid=ro, kspace=base[: co * m].numpy().reshape(co, m),
                          trajectory=tr.numpy(), trajectory_id=ro * 10000 + sp, pinned=True, out=out.numpy())
        r._keep = (tr, out)
        reqs.append(r)
    return reqs, base


def serve_pass(server, reqs, arrivals=None) -> dict:
    """Submit reqs (at the given arrival offsets in seconds, or all at once),
    wait for all, return the loop's statistics."""
    server.reset_stats()
    t0 = time.perf_counter()
    tickets = []
    for i, r in enumerate(reqs):
        if arrivals is not None:
            delay = t0 + arrivals[i] - time.perf_counter()
            if delay > 0:
                time.sleep(delay)
        tickets.append(server.submit(r))
    for t in tickets:
        server.wait(t, timeout_ms=120000)
    st = server.stats()
    st["samples_per_s"] = st["gridded_samples"] / st["wall_seconds"] if st["wall_seconds"] > 0 else None
    return st


def run_serve(args, n: int | None = None) -> dict:
    """The served stream: `n` requests through the request loop, once as the
    plain serial GPU path (one slot, batches of one request: each request is
    its own one-frame call) and once served (slots, ragged batches of up to
    --serve-batch requests), each as a burst (all submitted at once; the
    median of three bursts) and as Poisson arrivals at 90 % of the serial
    path's burst throughput."""
    import torch
    from kspacejet_gb300 import serve

    torch.cuda.init()
    n = n or args.serve_requests
    reqs, _base = serve_workload(n, seed=11)
    warm, _ = serve_workload(8, seed=12)
    samples = sum(r.kspace.size for r in reqs)
    # (name, slots, requests per batch, coil split); inputs are copied to the device in both
    modes = (("serial", 1, 1, 0), ("served", args.serve_slots, args.serve_batch, args.serve_coil_split))
    out = {"metric": "served gridded samples/s", "unit": "samples/s", "higher_is_better": True, "n_gpus": 1,
           "data": "synthetic", "dtype": "f32 (complex64 samples, float32 gridding/FFT)",
           "config": {"workload": "served stream of 2D radial slices (KB W=4, sigma=2, ramp DCF, RSS)",
                      "requests": n, "readout": list(SERVE_READOUTS), "spokes": [64, 805], "coils": [8, 32],
                      "gridded_samples": samples, "inputs": "pinned host memory, results to pinned host memory",
                      "serial": "1 slot, 1 request per call, inputs copied to the device",
                      "served": f"{args.serve_slots} slots, ragged batches of up to {args.serve_batch} requests "
                                f"(requests of at most {args.serve_coil_split} coils batched apart), inputs copied "
                                "to the device",
                      "device_memory_cap_gib": args.serve_cap_gib}}
    results = {}
    for name, slots, batch, split in modes:
        with serve.Server(slots=slots, device_memory_cap=args.serve_cap_gib << 30, max_batch_frames=batch,
                          coil_split=split) as s:
            serve_pass(s, warm)
            serve_pass(s, reqs)  # first pass uploads and caches the trajectories
            bursts = sorted((serve_pass(s, reqs) for _ in range(3)), key=lambda b: b["wall_seconds"])
            results[name] = {"burst": bursts[1]}  # the median of three bursts
    # Poisson arrivals at 90% of the serial path's burst throughput
    rate = 0.9 * n / results["serial"]["burst"]["wall_seconds"]
    rng = np.random.default_rng(13)
    arrivals = np.cumsum(rng.exponential(1.0 / rate, size=n))
    for name, slots, batch, split in modes:
        with serve.Server(slots=slots, device_memory_cap=args.serve_cap_gib << 30, max_batch_frames=batch,
                          coil_split=split) as s:
            serve_pass(s, warm)
            serve_pass(s, reqs)
            results[name]["poisson"] = serve_pass(s, reqs, arrivals)
    ser, srv = results["serial"], results["served"]
    out["value"] = srv["burst"]["samples_per_s"]
    out["serial_value"] = ser["burst"]["samples_per_s"]
    out["vs_serial"] = out["value"] / out["serial_value"]
    out["p50_ms"] = srv["poisson"]["latency_p50_ms"]
    out["p99_ms"] = srv["poisson"]["latency_p99_ms"]
    out["serial_p50_ms"] = ser["poisson"]["latency_p50_ms"]
    out["serial_p99_ms"] = ser["poisson"]["latency_p99_ms"]
    out["poisson_rate_per_s"] = rate
    out["results"] = results
    return out


# ------------------------------------------------ the other hot-path rows

def _warm(fn) -> None:
    """One call outside any timing: loads the call's kernels (lazy module
    loading) before the per-kernel event timing starts."""
    import torch

    fn()
    torch.cuda.synchronize()


def _time_gpu(fn, warmup: int, steps: int) -> float:
    """Mean ms per call of fn() over `steps` calls after `warmup`, CUDA events."""
    import torch

    for _ in range(warmup):
        fn()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        fn()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / steps


def run_rows(args) -> list[dict]:
    """One JSON line per remaining hot-path row, on the shapes of the
    configurations that use it (synthetic data of those shapes)."""
    import torch
    from kspacejet_gb300 import gpu, synth

    dev = torch.device("cuda", 0)
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    hbm = peaks.get("hbm_gbs", 6800.0)
    bf16 = peaks.get("bf16_tflops", 1900.0)
    w, s = max(args.warmup, 3), args.steps
    lines = []

    only = set(filter(None, (args.only or "").split(",")))

    def want(name: str) -> bool:
        return not only or name in only

    mm = 512 * 805
    rng = np.random.default_rng(3)
    L = gpu.lib()
    x = None
    if want("coil") or want("noise"):
        x = torch.from_numpy((rng.standard_normal((32, mm)) + 1j * rng.standard_normal((32, mm))).astype(np.complex64)).to(dev)
    g3, n3 = args.grid3, args.grid3 * 2 // 3

    if want("pipe_menon"):
        # Pipe-Menon density weights: the batched workload's trajectories (96 x 34 x 384, grid 384, W=4)
        traj = np.stack([synth.golden_angle_radial(READOUT, SPOKES, first_spoke=SPOKES * f) for f in range(FRAMES)])
        t = torch.from_numpy(traj).to(dev)
        _warm(lambda: gpu.pipe_menon_dcf(t, IMAGE, GRID, width=WIDTH, iterations=10))
        gpu.timing_reset()
        gpu.timing_enable(True)
        ms = _time_gpu(lambda: gpu.pipe_menon_dcf(t, IMAGE, GRID, width=WIDTH, iterations=10), w, s)
        kern = {n_: round(t_ / (w + s), 3) for n_, c_, t_ in gpu.timing_read()}  # ms per call
        gpu.timing_enable(False)
        m = traj.shape[0] * traj.shape[1]
        lines.append({"metric": "Pipe-Menon weights: sample-iterations/s", "value": m * 10 / (ms / 1e3),
                      "unit": "sample-iterations/s", "ms_per_call": ms, "dtype": "f64",
                      "config": {"workload": f"{FRAMES} frames x {SPOKES} spokes x {READOUT}, grid {GRID}, KB W={WIDTH}, "
                                             "10 iterations", "samples": m},
                      "kernels_ms_per_call": kern})

    if want("coil"):
        # coil covariance and compression: config 4 shape, 512 readout x 805 spokes, 32 -> 8 channels
        ws = torch.empty(gpu.lib().ksj_gpu_coil_covariance_workspace_bytes(32, mm), dtype=torch.uint8, device=dev)
        cov = torch.empty((32, 32), dtype=torch.complex64, device=dev)

        def covariance():
            gpu._check(L.ksj_gpu_coil_covariance(32, mm, x.data_ptr(), cov.data_ptr(), ws.data_ptr(), ws.numel(),
                                                 torch.cuda.current_stream().cuda_stream), "coil_covariance")

        _warm(covariance)
        gpu.timing_reset()
        gpu.timing_enable(True)
        ms = _time_gpu(covariance, w, s)
        kern = {n: (c, t_) for n, c, t_ in gpu.timing_read()}
        gpu.timing_enable(False)
        mma_ms = kern["k_cov_mma"][1] / kern["k_cov_mma"][0]
        kpad = (mm + 63) // 64 * 64
        tensor_flops = 2.0 * 128 * 64 * kpad  # one M=128 N=64 contraction over the padded samples
        lines.append({"metric": "coil covariance (tcgen05 split-BF16): samples/s", "value": mm / (ms / 1e3),
                      "unit": "samples/s", "ms_per_call": ms, "dtype": "bf16 x3 split, f32 accumulate",
                      "config": {"workload": "32 coils x 512 x 805 samples (complex64)"},
                      "kernels_ms": {k: round(v[1] / v[0], 4) for k, v in kern.items()},
                      "roofline": {"bound": "tensor", "kernel": "k_cov_mma",
                                   "achieved": round(tensor_flops / (mma_ms / 1e3) / 1e12, 2),
                                   "peak": bf16, "unit": "TFLOP/s", "frac": round(tensor_flops / (mma_ms / 1e3) / 1e12 / bf16, 4),
                                   "note": "the contraction is HBM-bound: 128 x 64 outputs per 64-sample tile"},
                      "hbm": {"bytes": 32 * mm * 8, "GBps": round(32 * mm * 8 / (ms / 1e3) / 1e9, 1),
                              "frac": round(32 * mm * 8 / (ms / 1e3) / 1e9 / hbm, 4)}})
        basis, _ = gpu.compression_basis(cov.cpu().numpy(), 8)
        bd = torch.from_numpy(basis).to(dev)
        y = torch.empty((8, mm), dtype=torch.complex64, device=dev)

        def compress():
            gpu._check(L.ksj_gpu_coil_compress(32, 8, mm, bd.data_ptr(), x.data_ptr(), y.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream), "coil_compress")

        ms = _time_gpu(compress, w, s)
        byts = (32 + 8) * mm * 8
        lines.append({"metric": "coil compression 32->8: samples/s", "value": mm / (ms / 1e3), "unit": "samples/s",
                      "ms_per_call": ms, "dtype": "f32",
                      "roofline": {"bound": "hbm", "achieved": round(byts / (ms / 1e3) / 1e9, 1), "peak": hbm,
                                   "unit": "GB/s", "frac": round(byts / (ms / 1e3) / 1e9 / hbm, 4)}})

    if want("noise"):
        # noise model from 32 x 65536 noise samples (covariance on the tensor cores, eigensolve on the
        # host) and prewhitening Y = W X of the same 32 x 412 160 k-space
        mn = 65536
        noise = torch.from_numpy((rng.standard_normal((32, mn)) + 1j * rng.standard_normal((32, mn))).astype(np.complex64)).to(dev)
        ms = _time_gpu(lambda: gpu.noise_model(noise), w, s)
        lines.append({"metric": "noise model estimate: noise samples/s", "value": mn / (ms / 1e3), "unit": "samples/s",
                      "ms_per_call": ms, "dtype": "bf16 x3 split covariance, f64 host eigensolve",
                      "config": {"workload": "32 coils x 65536 noise samples, whitening matrix to the device"}})
        wd = gpu.noise_model(noise)
        yw = torch.empty((32, mm), dtype=torch.complex64, device=dev)

        def prewhiten():
            gpu._check(L.ksj_gpu_noise_prewhiten(32, mm, wd.data_ptr(), x.data_ptr(), yw.data_ptr(),
                                                 torch.cuda.current_stream().cuda_stream), "noise_prewhiten")

        ms = _time_gpu(prewhiten, w, s)
        byts = 2 * 32 * mm * 8
        lines.append({"metric": "noise prewhitening 32x32: samples/s", "value": mm / (ms / 1e3), "unit": "samples/s",
                      "ms_per_call": ms, "dtype": "f32",
                      "config": {"workload": "32 coils x 512 x 805 samples (complex64)"},
                      "roofline": {"bound": "hbm", "achieved": round(byts / (ms / 1e3) / 1e9, 1), "peak": hbm,
                                   "unit": "GB/s", "frac": round(byts / (ms / 1e3) / 1e9 / hbm, 4)}})

    if want("kooshball") and args.spokes3 > 0:
        # 3-D kooshball: 256 readout x `spokes3` Fibonacci spokes, 20 coils, grid 384^3 (sigma 1.5), KB W=4,
        # |k|^2 density weights, RSS; complex64 and bf16 sample storage
        if args.spokes3 > 0:
            tr3 = torch.from_numpy(synth.kooshball(256, args.spokes3)).to(dev)
            m3 = tr3.shape[0]
            gen = torch.Generator(device=dev).manual_seed(5)
            k3 = torch.randn((20, m3), dtype=torch.complex64, device=dev, generator=gen)
            for fmt, name in ((gpu.SAMPLES_CF32, "complex64"), (gpu.SAMPLES_BF16, "bf16")):
                op3 = gpu.Gridding3(image=n3, grid=g3, channels=20, samples=m3, width=4, dcf=gpu.DCF_ANALYTIC_RAMP,
                                   output=gpu.OUTPUT_RSS, sample_format=fmt)
                kin = k3 if fmt == gpu.SAMPLES_CF32 else torch.stack([k3.real.to(torch.bfloat16),
                                                                      k3.imag.to(torch.bfloat16)], dim=-1).contiguous()
                ws3 = op3.new_workspace(dev)
                o3 = op3.new_output(dev)
                _warm(lambda: op3.run(kin, tr3, o3, ws3))
                gpu.timing_reset()
                gpu.timing_enable(True)
                reps3 = max(1, min(s, 3))
                ms = _time_gpu(lambda: op3.run(kin, tr3, o3, ws3), 1, reps3)
                kern = {n_: round(t_ / (1 + reps3), 3) for n_, c_, t_ in gpu.timing_read()}  # ms per call
                gpu.timing_enable(False)
                lines.append({"metric": "3-D kooshball gridded samples/s", "value": 20 * m3 / (ms / 1e3),
                              "unit": "samples/s", "ms_per_call": ms, "dtype": f"f32 ({name} sample storage)",
                              "config": {"workload": f"256 x {args.spokes3} spokes kooshball, 20 coils, grid {g3}^3, "
                                                     "KB W=4, sigma 1.5, |k|^2 DCF, RSS", "gridded_samples": 20 * m3,
                                         "workspace_bytes": ws3.numel()},
                              "kernels_ms_per_call": kern})
                del ws3, o3
            # 3-D Pipe-Menon weights for the same trajectory (FP64, 10 iterations)
            _warm(lambda: gpu.pipe_menon_dcf3(tr3, n3, g3, width=4, iterations=10))
            gpu.timing_reset()
            gpu.timing_enable(True)
            calls = 1 + max(1, min(s, 3))
            ms = _time_gpu(lambda: gpu.pipe_menon_dcf3(tr3, n3, g3, width=4, iterations=10), 1, calls - 1)
            kern = {n_: round(t_ / calls, 3) for n_, c_, t_ in gpu.timing_read()}  # ms per call
            gpu.timing_enable(False)
            lines.append({"metric": "3-D Pipe-Menon weights: sample-iterations/s", "value": m3 * 10 / (ms / 1e3),
                          "unit": "sample-iterations/s", "ms_per_call": ms, "dtype": "f64",
                          "config": {"workload": f"256 x {args.spokes3} spokes kooshball, grid {g3}^3, KB W=4, "
                                                 "10 iterations", "samples": m3},
                          "kernels_ms_per_call": kern})

    if want("direct_forward"):
        # exact direct forward NUDFT (the reference's nufft2_forward on its Eigen backend): 128^2 image,
        # 8 coils, 34 spokes x 256 readout
        imf = torch.from_numpy((rng.standard_normal((128, 128, 8)) + 1j * rng.standard_normal((128, 128, 8))).astype(np.complex64)).to(dev)
        trf = torch.from_numpy(synth.golden_angle_radial(256, 34)).to(dev)
        ms = _time_gpu(lambda: gpu.direct_forward(imf, trf), 1, max(1, min(s, 5)))
        pairs = 128 * 128 * trf.shape[0]
        lines.append({"metric": "direct forward NUDFT: (sample, pixel) pairs/s", "value": pairs / (ms / 1e3),
                      "unit": "pairs/s", "ms_per_call": ms, "dtype": "f32 (exact phase per pair)",
                      "config": {"workload": "128 x 128 image, 8 coils, 34 x 256 golden-angle samples",
                                 "complex_macs": pairs * 8}})

    if want("kb_forward"):
        # Kaiser-Bessel forward NUFFT on the batched shape: 96 frames of 192^2 x 32 coil images -> 34 x 384 samples
        trh, _ = make_inputs()
        trk = torch.from_numpy(trh).to(dev)
        fop = gpu.kb_gridding(image=IMAGE, grid=GRID, channels=COILS, samples=trh.shape[1], frames=FRAMES, width=WIDTH,
                              dcf=gpu.DCF_NONE, output=gpu.OUTPUT_COIL_LAST)
        fimg = torch.randn((FRAMES, IMAGE, IMAGE, COILS), dtype=torch.complex64, device=dev)
        fws = torch.empty(fop.forward_workspace_bytes(), dtype=torch.uint8, device=dev)
        _warm(lambda: fop.forward(fimg, trk, fws))
        gpu.timing_reset()
        gpu.timing_enable(True)
        ms = _time_gpu(lambda: fop.forward(fimg, trk, fws), w, s)
        kern = {n_: round(t_ / c_, 4) for n_, c_, t_ in gpu.timing_read()}
        gpu.timing_enable(False)
        lines.append({"metric": "Kaiser-Bessel forward NUFFT: samples/s", "value": FRAMES * COILS * trh.shape[1] / (ms / 1e3),
                      "unit": "samples/s", "ms_per_call": ms, "dtype": "f32",
                      "config": {"workload": f"{FRAMES} frames x {COILS} coils, {IMAGE}^2 images -> {SPOKES} x {READOUT} "
                                             f"samples per frame, KB W={WIDTH}, grid {GRID}"},
                      "kernels_ms": kern})
        del fimg, fws

    if want("cartesian"):
        # Cartesian coil images: 8 frames x 32 coils x 256 x 256, coil-last output
        kc = torch.from_numpy((rng.standard_normal((8, 32, 256, 256)) + 1j * rng.standard_normal((8, 32, 256, 256))).astype(np.complex64)).to(dev)
        ms = _time_gpu(lambda: gpu.cartesian_ifft2(kc), w, s)
        byts = 2 * kc.numel() * 8  # k-space read, coil-last images written
        lines.append({"metric": "Cartesian coil images: images/s", "value": 8 * 32 / (ms / 1e3), "unit": "images/s",
                      "ms_per_call": ms, "dtype": "f32",
                      "config": {"workload": "8 frames x 32 coils x 256 x 256, inverse 2-D DFT, coil-last"},
                      "roofline": {"bound": "hbm", "achieved": round(byts / (ms / 1e3) / 1e9, 1), "peak": hbm,
                                   "unit": "GB/s", "frac": round(byts / (ms / 1e3) / 1e9 / hbm, 4),
                                   "note": "algorithmic bytes = k-space in + images out; the "
                                           "row-transformed intermediate adds 2 more passes"}})
        del kc

    if want("combine"):
        # Walsh 7x7 on the compressed 8-coil image (256 x 256), and RSS of 32 coils
        img = torch.from_numpy((rng.standard_normal((256, 256, 8)) + 1j * rng.standard_normal((256, 256, 8))).astype(np.complex64)).to(dev)
        ms = _time_gpu(lambda: gpu.walsh_combine(img, window=7, iterations=24), w, s)
        lines.append({"metric": "Walsh 7x7 combine: pixels/s", "value": 256 * 256 / (ms / 1e3), "unit": "pixels/s",
                      "ms_per_call": ms, "dtype": "f32", "config": {"workload": "256 x 256 x 8 coils, 24 power iterations"}})
        img32 = torch.from_numpy((rng.standard_normal((256, 256, 32)) + 1j * rng.standard_normal((256, 256, 32))).astype(np.complex64)).to(dev)
        ms = _time_gpu(lambda: gpu.rss_coil_last(img32), w, s)
        byts = 256 * 256 * (32 * 8 + 4)
        lines.append({"metric": "RSS combine: pixels/s", "value": 256 * 256 / (ms / 1e3), "unit": "pixels/s",
                      "ms_per_call": ms, "dtype": "f32",
                      "roofline": {"bound": "hbm", "achieved": round(byts / (ms / 1e3) / 1e9, 1), "peak": hbm,
                                   "unit": "GB/s", "frac": round(byts / (ms / 1e3) / 1e9 / hbm, 4)}})
    return lines


def main() -> int:
    global FRAMES
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--frames", type=int, default=FRAMES,
                    help="frames per call (default: the 96-frame workload; fewer only for small profiling cases)")
    ap.add_argument("--tuning", default="",
                    help="fixed gridding tuning cg,cb,fpp,rb,parts[,column_pass] instead of the autotuner")
    ap.add_argument("--serve", action="store_true", help="served-stream benchmark (separate JSON line)")
    ap.add_argument("--rows", action="store_true", help="the other hot-path rows (one JSON line each)")
    ap.add_argument("--spokes3", type=int, default=40000, help="--rows: spokes of the 3-D kooshball (0 skips it)")
    ap.add_argument("--grid3", type=int, default=384, help="--rows: grid of the 3-D kooshball (image = 2/3 of it)")
    ap.add_argument("--only", default="", help="--rows: a comma list of rows to run (pipe_menon, coil, noise, "
                                               "kooshball, direct_forward, kb_forward, cartesian, combine)")
    ap.add_argument("--skip-extra", action="store_true",
                    help="skip the width-6 and drop-in legs (small profiling runs)")
    ap.add_argument("--serve-requests", type=int, default=160)
    ap.add_argument("--serve-slots", type=int, default=2)
    ap.add_argument("--serve-batch", type=int, default=32, help="requests per ragged batch of the served path")
    ap.add_argument("--serve-cap-gib", type=int, default=64)
    ap.add_argument("--serve-coil-split", type=int, default=16,
                    help="served path: requests of at most this many coils form their own batches (0: no split)")
    args = ap.parse_args()
    FRAMES = args.frames
    if args.warmup < 3 and args.impl == "ours":
        args.warmup = 3
    if args.rows:
        import kspacejet_gb300

        kspacejet_gb300.build()
        for line in run_rows(args):
            print(json.dumps(line))
        return 0
    if args.serve:
        import kspacejet_gb300

        kspacejet_gb300.build()
        res = run_serve(args)
    elif args.impl == "reference":
        res = run_reference(args)
    else:
        import kspacejet_gb300

        kspacejet_gb300.build()
        res = run_ours(args)
    if res is not None:
        print(json.dumps(res))
    return 0


if __name__ == "__main__":
    sys.exit(main())
