#!/usr/bin/env python
"""Benchmark: plane integrals/s of the grid-sampled 3D Radon transform at 128^3.

Workload (one "step"): the forward Radon transform of a 128^3 volume (sum of
16 seeded ellipsoids, seed 1001) on the Gauss-uniform sphere grid of 64
latitudes x 128 longitudes x 256 shifts = 2,097,152 plane integrals, each the
reference's lattice (step 1/n) restricted to [-n, n)^2 = 256 x 256 points with
the trilinear sampler (radon_grid/src/integral.c:26-58 with
cube_trilinear_interp).  Synthetic data, generated here.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Prints one JSON line (rank 0).  ``value`` is device-timed throughput with the
volume resident in HBM (CUDA events on the library's stream, L2 flushed before
every timed step); ``e2e`` is the same metric through the public API with the
FP64 host volume copied in from pinned memory and the FP64 results copied
back every step.  ``--impl reference`` times the reference's own C code
(oracle/_ref, compiled from the reference sources) on the host cores.
With N > 1 every rank runs the whole workload on its own GPU (independent
replicas, weak scaling); time is the maximum over ranks.
"""
from __future__ import annotations

import argparse
import importlib.util
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
PKG_DIR = ROOT / "wrt-project_b200"

N, ELLIPSOIDS, SEED = 128, 16, 1001
NPHI, NTHETA, NSHIFT = 128, 64, 256
HALF_EXTENT = N  # lattice [-n, n)^2 -> 256 x 256 samples per plane
BYTES_PER_SAMPLE = 32  # eight FP32 voxel reads per trilinear sample
# the headline metric's name as the benchmark's specification states it; the
# workload itself (sphere grid, shifts, sampler, lattice) is spelled out in
# each line's "config"
METRIC = "plane integrals/s @128³ (served vs plain, same B200, rel.err≤1e-5); p50/p99 ms"
UNIT = "plane integrals/s"


def load_package():
    spec = importlib.util.spec_from_file_location(
        "wrt_b200", PKG_DIR / "__init__.py", submodule_search_locations=[str(PKG_DIR)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["wrt_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# ------------------------------------------------------------ distributed
class Dist:
    def __init__(self, gpus: int):
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local_rank = int(os.environ.get("LOCAL_RANK", "0"))
        self.pg = None
        if self.world > 1:
            import datetime

            import torch.distributed as dist

            dist.init_process_group("gloo", timeout=datetime.timedelta(seconds=300))
            self.pg = dist

    def barrier(self):
        if self.pg:
            self.pg.barrier()

    def max(self, x: float) -> float:
        if not self.pg:
            return x
        import torch

        t = torch.tensor([x], dtype=torch.float64)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def close(self):
        if self.pg:
            self.pg.destroy_process_group()


# ------------------------------------------------------------ clocks
class ClockSampler:
    """nvidia-smi samples every 200 ms while the timed region runs."""

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device, self.proc, self.lines = device, None, []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-i", str(self.device), "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self) -> dict:
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.thread.join(timeout=2)
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 7:
                continue
            try:
                sm.append(float(parts[0]))
                smax = float(parts[1])
            except ValueError:
                continue
            for nm, v in zip(names, parts[3:7]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(sm)}


# ------------------------------------------------------------ CPU baselines
def cpu_threads() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def plane_sample(count: int, seed: int):
    """A seeded random subset of the workload's planes (phi, theta, shift)."""
    sys.path.insert(0, str(ROOT))
    import oracle as O

    phi, theta, _, shift = O.radon_grid(NPHI, NTHETA, NSHIFT)
    rng = np.random.default_rng(seed)
    idx = rng.integers(0, NPHI * NTHETA * NSHIFT, size=count)
    it, ip, i_s = idx % NTHETA, (idx // NTHETA) % NPHI, idx // (NTHETA * NPHI)
    return phi[ip], theta[it], shift[i_s]


def time_reference_planes(vol, count, seed, threads):
    """The reference's plane_integral (nearest sampler, lattice [-2n,2n)^2, as
    shipped in radon_grid) over `count` sampled planes; returns planes/s."""
    sys.path.insert(0, str(ROOT))
    import oracle as O

    ref = O.Reference()
    p, t, s = plane_sample(count, seed)
    t0 = time.perf_counter()
    ref.plane_integrals(vol, p, t, s, nthreads=threads)
    return count / (time.perf_counter() - t0)


def cpu_baseline(vol, budget_s=12.0):
    threads = cpu_threads()
    sys.path.insert(0, str(ROOT))
    import oracle as O

    if not O.Reference.available():
        return {"value": None, "unit": UNIT, "cores": threads, "kind": "reference",
                "sample": "oracle/_ref not built"}
    # calibrate on a small sample, then size the measured sample to ~budget_s
    rate = time_reference_planes(vol, 256, 1, threads)
    count = int(max(512, min(200000, rate * budget_s)))
    rate = time_reference_planes(vol, count, 2, threads)
    # the FP64 restatement with the benchmark's own sampler and lattice
    p, t, s = plane_sample(max(256, count // 8), 3)
    t0 = time.perf_counter()
    O.radon_planes(vol, p, t, s, sampler=O.TRILINEAR, half_extent=HALF_EXTENT, nthreads=threads)
    port_rate = len(p) / (time.perf_counter() - t0)
    return {"value": rate, "unit": UNIT, "cores": threads, "kind": "reference",
            "sample": f"{count} seeded random planes of the 128^3 workload; the reference's "
                      f"radon_grid plane_integral as shipped (nearest sampler, 512^2 lattice, "
                      f"FP64), gcc -O2, OpenMP over planes",
            "port_trilinear": {"value": port_rate, "unit": UNIT, "kind": "port",
                               "sample": f"{len(p)} planes, the benchmark's own definition "
                                         f"(trilinear, 256^2 lattice), FP64 oracle restatement"}}


def run_reference(args, dist):
    if dist.rank != 0:
        return 0
    sys.path.insert(0, str(PKG_DIR))
    from phantom import ellipsoid_phantom
    sys.path.insert(0, str(ROOT))
    import oracle as O

    threads = cpu_threads()
    if not O.Reference.available():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref not built "
                          "(reference sources were not present at build time)"}))
        return 0
    vol = ellipsoid_phantom(N, ELLIPSOIDS, SEED)
    per_step = int(os.environ.get("WRT_REF_PLANES_PER_STEP", "2048"))
    for w in range(args.warmup):
        time_reference_planes(vol, per_step, 100 + w, threads)
    t_total = 0.0
    for k in range(args.steps):
        t0 = time.perf_counter()
        time_reference_planes(vol, per_step, 1000 + k, threads)
        t_total += time.perf_counter() - t0
    value = per_step * args.steps / t_total
    ms_per_step = 1e3 * t_total / args.steps
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic",
        "config": {"workload": "radon_grid 128^3, 64x128x256 planes", "n": N,
                   "sphere_grid": [NTHETA, NPHI], "shifts": NSHIFT,
                   "per_step": f"{per_step} seeded random planes of the workload"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "reference",
                         "sample": f"{per_step} planes per step; radon_grid plane_integral as "
                                   f"shipped (nearest sampler, 512^2 lattice), FP64"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


# ------------------------------------------------------------ the other hot paths
RAY_SLICES, RAY_SHIFTS, RAY_PHIS = 128, 128, 128


def rotated_frame(seed):
    rng = np.random.default_rng(seed)
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    frame = q * np.sign(np.diag(r))
    if np.linalg.det(frame) < 0:
        frame[:, 0] = -frame[:, 0]
    return frame


def timed_device_calls(ctx, call, steps, warmup):
    """CUDA-event times (ms) of `call` on the library's stream, L2 flushed
    before each timed call."""
    for _ in range(max(warmup, 3)):
        call()
    ctx.synchronize()
    times = []
    for _ in range(steps):
        ctx.flush_l2()
        ctx.timer_start()
        call()
        times.append(ctx.timer_stop())
    return times


def other_paths(wrt, ctx, phantom, steps, warmup, smem_bw, hbm_peak, with_cpu):
    """The ray transform (reference frame and one rotated frame), the
    reduction of ray data to Radon data, and the backprojection, at 128^3,
    through their device-resident entry points: device time per call, units/s,
    a roofline -- where every counted sample is read on its own, its bytes against
    the measured shared-memory/L1 bandwidth; where samples share what is read, the
    compulsory HBM bytes, with the samples' figure beside it -- and, in the CPU leg, the
    reference's own code on a bounded seeded sample of the same units, timed
    on the host cores and compared with the GPU's values there."""
    n = N
    vol = wrt.Volume(ctx, n)
    vol.upload(phantom.astype(np.float32))
    grid = wrt.Grid(ctx, NPHI, NTHETA, NSHIFT)
    nrays = RAY_SLICES * RAY_SHIFTS * RAY_PHIS
    rays_d = wrt.DeviceBuffer(ctx, nrays * 8)
    radon_d = wrt.DeviceBuffer(ctx, grid.nplanes * 8)
    adj_d = wrt.DeviceBuffer(ctx, n ** 3 * 8)
    frame = rotated_frame(SEED)
    rng = np.random.default_rng(SEED + 7)
    gauss = rng.standard_normal((NSHIFT, NPHI, NTHETA))
    res = {}

    def counted(call):
        ctx.count_samples(True)
        call()
        c = ctx.sample_count()
        ctx.count_samples(False)
        return c

    def entry(name, call, units, unit, bytes_per_sample, samples, sample_unit, download,
              shared_hbm=None):
        times = timed_device_calls(ctx, call, steps, warmup)
        ms = statistics.mean(times)
        gather = {"achieved": samples * bytes_per_sample / (ms * 1e-3) / 1e9, "peak": smem_bw / 1e9,
                  "unit": "GB/s", "algorithmic_bytes": f"{bytes_per_sample} B per {sample_unit}",
                  "samples_per_call": samples}
        if shared_hbm is None:
            roof = {"bound": "l1tex", **gather, "frac": gather["achieved"] / gather["peak"]}
        else:
            achieved = shared_hbm / (ms * 1e-3) / 1e9
            roof = {"bound": "latency", "achieved": achieved, "peak": hbm_peak, "unit": "GB/s",
                    "frac": achieved / hbm_peak,
                    "note": "compulsory HBM bytes (inputs once, results once)",
                    "samples": {**gather, "note": "what reading every sample on its own would take; "
                                                  "samples share what is read, so no roofline"}}
        res[name] = {"value": units / (ms * 1e-3), "unit": unit, "ms_per_call": ms,
                     "ms_median": statistics.median(times), "gpu_launches_per_call": None,
                     "roofline": roof}
        return download()

    ray_call = lambda fr=None: wrt.ray_forward_device(ctx, vol, RAY_SLICES, RAY_SHIFTS, RAY_PHIS,
                                                       rays_d.ptr, frame=fr)
    dl_rays = lambda: rays_d.download(np.empty((RAY_SLICES, RAY_SHIFTS, RAY_PHIS)))
    l0 = ctx.launches
    rays = entry("ray", ray_call, nrays, "rays/s", BYTES_PER_SAMPLE, counted(ray_call),
                 "trilinear sample (8 FP32 corners)", dl_rays, shared_hbm=4 * n ** 3 + 8 * nrays)
    res["ray"]["gpu_launches_per_call"] = (ctx.launches - l0) // (steps + max(warmup, 3) + 1)
    rc = lambda: ray_call(frame)
    rays_rot = entry("ray_rotated", rc, nrays, "rays/s", BYTES_PER_SAMPLE, counted(rc),
                     "trilinear sample (8 FP32 corners)", dl_rays)
    # the reduction reads the reference-frame rays (128 offsets) from the device
    ray_call()
    red = lambda: wrt.radon_reduction_device(ctx, rays_d.ptr, n, RAY_SHIFTS, grid, radon_d.ptr)
    radon = entry("reduction", red, grid.nplanes, "plane integrals/s", 48, counted(red),
                  "slice sample (6 shared loads of 8 B)",
                  lambda: radon_d.download(np.empty((NSHIFT, NPHI, NTHETA))))
    gauss_d = wrt.DeviceBuffer(ctx, gauss.nbytes)
    gauss_d.upload(gauss)
    adj = lambda: wrt.radon3d_adjoint_device(ctx, gauss_d.ptr, grid, n, adj_d.ptr)
    evals = n ** 3 * NPHI * NTHETA
    adjoint = entry("adjoint", adj, n ** 3, "voxels/s", 16, evals,
                    "spline evaluation (one 16 B record)",
                    lambda: adj_d.download(np.empty((n, n, n))),
                    shared_hbm=8 * grid.nplanes + 8 * n ** 3)
    # the reference's default sampler: nearest cell on the 4n x 4n lattice
    near = lambda: wrt.radon_forward_device(ctx, vol, grid, radon_d.ptr, sampler=wrt.NEAREST)
    nearest = entry("nearest", near, grid.nplanes, "plane integrals/s", 4, counted(near),
                    "nearest sample (one FP32 cell value)",
                    lambda: radon_d.download(np.empty((NSHIFT, NPHI, NTHETA))),
                    shared_hbm=4 * n ** 3 + 8 * grid.nplanes)
    plain_near = lambda: wrt.radon_forward_device(ctx, vol, grid, radon_d.ptr, sampler=wrt.NEAREST,
                                                  kernel=wrt.KERNEL_PLAIN)
    pt = timed_device_calls(ctx, plain_near, 2, 1)
    res["nearest"]["plain_kernel_ms"] = statistics.mean(pt)
    res["nearest"]["over_plain"] = statistics.mean(pt) / res["nearest"]["ms_per_call"]
    for k, w in (("nearest", "128^3, 64x128 sphere grid x 256 shifts, nearest sampler, lattice "
                             "[-2n, 2n)^2 with step 1/n (radon_grid's defaults)"),
                 ("ray", "128^3, 128 layers x 128 shifts x 128 angles, reference frame"),
                 ("ray_rotated", "the same in one seeded rotated layer frame"),
                 ("reduction", "128^3 rays (128 offsets) -> 64x128 sphere grid x 256 shifts"),
                 ("adjoint", "N(0,1) Radon data 64x128x256 -> 128^3 voxels")):
        res[k]["workload"] = w
    # what binds each kernel, from its committed ncu capture (a profiler cannot
    # run inside the timed bench): the byte figure above is the algorithmic
    # gather, not always the limit
    cap = "(profiles/table_kernels_128cubed.md)"
    for k, b in (("nearest", "gathers of the row tables with few warps resident, late blocks of "
                             f"dependent launches {cap}"),
                 ("ray", f"L1: 87 % of its throughput, column loads along z {cap}"),
                 ("ray_rotated", "L1 gathers: 82 % of L1 throughput "
                                 "(profiles/ray_kernel_128cubed.md)"),
                 ("reduction", f"shared-memory wavefronts: 90 % of the peak {cap}"),
                 ("adjoint", f"record gathers: L1 at 81 % on the SMs that are busy {cap}")):
        res[k]["roofline"]["limit_measured"] = b
    if with_cpu:
        import oracle as O
        cores = cpu_threads()
        ref = O.Reference() if O.Reference.available() else None
        s_grid, phi_grid = O.ray_grid(RAY_SHIFTS, RAY_PHIS)
        # nearest: the reference's own plane_integral (its default sampler) on
        # 1024 seeded planes
        if ref:
            m = 1024
            idx = rng.integers(0, grid.nplanes, size=m)
            it, ip, i_s = idx % NTHETA, (idx // NTHETA) % NPHI, idx // (NTHETA * NPHI)
            phi, theta, _, shift = O.radon_grid(NPHI, NTHETA, NSHIFT)
            t0 = time.perf_counter()
            got = ref.plane_integrals(phantom, phi[ip], theta[it], shift[i_s], cores)
            wall = time.perf_counter() - t0
            res["nearest"]["cpu_baseline"] = {
                "value": m / wall, "unit": "plane integrals/s", "cores": cores,
                "kind": "reference",
                "sample": f"{m} seeded planes, radon_grid's plane_integral (oracle/_ref), FP64"}
            res["nearest"]["rel_l2_vs_reference_on_sample"] = float(
                np.linalg.norm(nearest.reshape(-1)[idx] - got) / np.linalg.norm(got))
        # ray: the reference's ray_transform on 16384 seeded rays
        m = 16384
        idx = rng.integers(0, nrays, size=m)
        iz, i_s, ip = idx // (RAY_SHIFTS * RAY_PHIS), (idx // RAY_PHIS) % RAY_SHIFTS, idx % RAY_PHIS
        z = -1.0 + iz * (2.0 / (RAY_SLICES - 1))
        if ref:
            t0 = time.perf_counter()
            got = ref.rays(phantom, z, s_grid[i_s], phi_grid[ip], cores)
            wall = time.perf_counter() - t0
            res["ray"]["cpu_baseline"] = {
                "value": m / wall, "unit": "rays/s", "cores": cores, "kind": "reference",
                "sample": f"{m} seeded rays, ray_grid's ray_transform (oracle/_ref), FP64"}
            res["ray"]["rel_l2_vs_reference_on_sample"] = float(
                np.linalg.norm(rays.reshape(-1)[idx] - got) / np.linalg.norm(got))
        # rotated frame: the FP64 restatement (the reference has no layer frames)
        m = 1024
        idx = idx[:m]
        t0 = time.perf_counter()
        got = np.array([O.ray_transform(phantom, a, s_grid[b], phi_grid[c], frame=frame)
                        for a, b, c in zip(z[:m], i_s[:m], ip[:m])])
        wall = time.perf_counter() - t0
        res["ray_rotated"]["cpu_baseline"] = {
            "value": m / wall, "unit": "rays/s", "cores": 1, "kind": "port",
            "sample": f"{m} seeded rays, FP64 oracle restatement with the frame, one thread"}
        res["ray_rotated"]["rel_l2_vs_oracle_on_sample"] = float(
            np.linalg.norm(rays_rot.reshape(-1)[idx] - got) / np.linalg.norm(got))
        # reduction: the restatement on 2048 seeded planes (decoupled shift grids);
        # the reference itself on coupled grids (its own definition) for the timing
        m = 2048
        sel = rng.integers(0, [NSHIFT, NPHI, NTHETA], size=(m, 3))
        got = O.reduction_planes(rays[:n], NSHIFT, NTHETA, sel[:, 0], sel[:, 1], sel[:, 2],
                                 nthreads=cores)
        res["reduction"]["rel_l2_vs_oracle_on_sample"] = float(
            np.linalg.norm(radon[sel[:, 0], sel[:, 1], sel[:, 2]] - got) / np.linalg.norm(got))
        if ref:
            rays_c = ctx.ray_grid(phantom, n, NSHIFT, RAY_PHIS)
            t0 = time.perf_counter()
            ref.reduction_planes(rays_c, NTHETA, sel[:, 0], sel[:, 1], sel[:, 2], cores)
            wall = time.perf_counter() - t0
            res["reduction"]["cpu_baseline"] = {
                "value": m / wall, "unit": "plane integrals/s", "cores": cores,
                "kind": "reference",
                "sample": f"{m} seeded planes, radon_reduction's radon_reduction (oracle/_ref) "
                          "on rays with 256 offsets (the reference couples the shift grids)"}
        # adjoint: the reference's radon3d_adjoint at 128 seeded voxels
        m = 128
        idx = rng.integers(0, n ** 3, size=m)
        a, b, c = idx // (n * n), (idx // n) % n, idx % n  # [iz][ix][iy]
        ctr = lambda i: -1.0 + (2.0 * i + 1.0) / n
        if ref:
            t0 = time.perf_counter()
            got = ref.adjoint_points(gauss, ctr(b), ctr(c), ctr(a), cores)
            wall = time.perf_counter() - t0
            res["adjoint"]["cpu_baseline"] = {
                "value": m / wall, "unit": "voxels/s", "cores": cores, "kind": "reference",
                "sample": f"{m} seeded voxels, the backprojection's radon3d_adjoint (oracle/_ref)"}
            res["adjoint"]["rel_l2_vs_reference_on_sample"] = float(
                np.linalg.norm(adjoint.reshape(-1)[idx] - got) / np.linalg.norm(got))
    for b in (rays_d, radon_d, adj_d, gauss_d):
        b.close()
    grid.close()
    vol.close()
    return res


def config_runs(wrt, ctx, steps):
    """The ray and 256^3 configurations at their stated sizes through the
    device-resident entry points (device time, CUDA events on the library's
    stream, L2 flushed before each timed call): the ray transform in 64 layer
    orientations (the reference frame and 63 seeded rotations) x 128 layers x
    128 shifts x 128 angles at 128^3 followed by the reduction of the reference
    frame's rays to a 64x128 sphere grid x 256 shifts; the forward transform
    of a 256^3 volume (16 seeded ellipsoids) in FP32 and in BF16 storage on a
    96x192 sphere grid x 384 shifts (trilinear, lattice [-n, n)^2); and the
    backprojection of seeded N(0,1) Radon data on that grid back to 256^3."""
    from wrt_b200.phantom import ellipsoid_phantom, layer_frames

    res = {}
    n = 128
    vol = wrt.Volume(ctx, n)
    vol.upload(ellipsoid_phantom(n, ELLIPSOIDS, SEED).astype(np.float32))
    frames = layer_frames(64, 1101)
    nrays = n * RAY_SHIFTS * RAY_PHIS
    rays0 = wrt.DeviceBuffer(ctx, nrays * 8)
    rays = wrt.DeviceBuffer(ctx, nrays * 8)
    grid = wrt.Grid(ctx, NPHI, NTHETA, NSHIFT)
    radon = wrt.DeviceBuffer(ctx, grid.nplanes * 8)

    def rays_and_reduction():
        for k, F in enumerate(frames):
            wrt.ray_forward_device(ctx, vol, n, RAY_SHIFTS, RAY_PHIS,
                                   (rays0 if k == 0 else rays).ptr, frame=None if k == 0 else F)
        wrt.radon_reduction_device(ctx, rays0.ptr, n, RAY_SHIFTS, grid, radon.ptr)
    t = statistics.mean(timed_device_calls(ctx, rays_and_reduction, steps, 1))
    res["rays_64_orientations_and_reduction_128"] = {
        "ms": t, "rays_per_s": 64 * nrays / (t * 1e-3),
        "workload": "128^3: ray transform in 64 layer orientations x 128 layers x 128 shifts x "
                    "128 angles, then the reduction of orientation 0 to 64x128 x 256 shifts"}
    for b in (rays0, rays, radon):
        b.close()
    grid.close()
    vol.close()

    n3, nphi, ntheta, nshift = 256, 192, 96, 384
    phantom = ellipsoid_phantom(n3, ELLIPSOIDS, 1003)
    grid3 = wrt.Grid(ctx, nphi, ntheta, nshift)
    out3 = wrt.DeviceBuffer(ctx, grid3.nplanes * 8)
    for storage, name in ((wrt.STORAGE_F32, "forward_256_f32"),
                          (wrt.STORAGE_BF16, "forward_256_bf16")):
        v = wrt.Volume(ctx, n3, storage=storage)
        v.upload(phantom)
        t = statistics.mean(timed_device_calls(
            ctx, lambda: wrt.radon_forward_batch(ctx, [(v, grid3, out3.ptr, n3)]), steps, 1))
        res[name] = {"ms": t, "plane_integrals_per_s": grid3.nplanes / (t * 1e-3),
                     "workload": f"256^3 ({'FP32' if storage == wrt.STORAGE_F32 else 'BF16'} "
                                 "storage), 96x192 sphere grid x 384 shifts, trilinear, "
                                 "lattice [-n, n)^2"}
        v.close()
    g = np.random.default_rng(4004).standard_normal((nshift, nphi, ntheta))
    out3.upload(g)
    adj = wrt.DeviceBuffer(ctx, n3 ** 3 * 8)
    t = statistics.mean(timed_device_calls(
        ctx, lambda: wrt.radon3d_adjoint_device(ctx, out3.ptr, grid3, n3, adj.ptr), steps, 1))
    res["adjoint_256"] = {"ms": t, "voxels_per_s": n3 ** 3 / (t * 1e-3),
                          "spline_evaluations_per_s": n3 ** 3 * nphi * ntheta / (t * 1e-3),
                          "workload": "N(0,1) Radon data 96x192 x 384 shifts -> 256^3 voxels"}
    adj.close()
    out3.close()
    grid3.close()
    return res


def batch_vs_one_per_launch(wrt, ctx, steps, count=64, edges=(48, 64, 96, 128, 160, 192),
                            lat=(16, 97), shifts=(64, 257), seed=2002):
    """`count` FP32 volumes of uneven edge lengths (drawn from `edges`), each
    with its own sphere grid (lat latitudes x twice as many longitudes,
    `shifts` shifts; half-open ranges): all in ONE graph-captured launch of the
    persistent kernel (wrt_radon_forward_batch) against the same requests run
    one wrt_radon_forward_device call (staged kernel) per request.  Device time
    with CUDA events, L2 flushed before each timed run.  The default is the
    batched configuration (64 requests, n = 48..192); with small requests
    (n = 16..48) a single request cannot fill the GPU, which is where one
    launch for all of them pays."""
    from wrt_b200.phantom import ellipsoid_phantom

    rng = np.random.default_rng(seed)
    reqs, keep, planes = [], [], 0
    for k in range(count):
        n = int(rng.choice(list(edges)))
        nth = int(rng.integers(*lat))
        ns = int(rng.integers(*shifts))
        v = wrt.Volume(ctx, n)
        v.upload(ellipsoid_phantom(n, int(rng.integers(4, 25)), 3000 + k).astype(np.float32))
        g = wrt.Grid(ctx, 2 * nth, nth, ns)
        out = wrt.DeviceBuffer(ctx, g.nplanes * 8)
        reqs.append((v, g, out.ptr, n))
        keep.append((v, g, out))
        planes += g.nplanes
    batched = lambda: wrt.radon_forward_batch(ctx, reqs)

    def one_by_one():
        for v, g, ptr, n in reqs:
            wrt.radon_forward_device(ctx, v, g, ptr, sampler=wrt.TRILINEAR, half_extent=n,
                                     kernel=wrt.KERNEL_STAGED)
    tb = timed_device_calls(ctx, batched, steps, 2)
    first = [o.download(np.empty(g.nplanes)) for _, g, o in keep]
    to = timed_device_calls(ctx, one_by_one, steps, 2)
    same = all(np.array_equal(f, o.download(np.empty(g.nplanes)))
               for f, (_, g, o) in zip(first, keep))
    for v, g, o in keep:
        o.close(); g.close(); v.close()
    mb, mo = statistics.mean(tb), statistics.mean(to)
    return {"requests": count, "edges": sorted(set(int(r[3]) for r in reqs)),
            "planes": planes, "batched_ms": mb, "one_per_launch_ms": mo,
            "ratio": mo / mb, "batched_plane_integrals_per_s": planes / (mb * 1e-3),
            "results_bitwise_equal": same,
            "note": f"ratio = time of {count} single-request launches / time of one batched launch"}


# ------------------------------------------------------------ our arm
def served_stream(wrt, srv, pin_vol, pin_outs, steps):
    """K requests of the workload through the serving loop, each with its FP32
    volume in pinned host memory and its FP64 result copied back to pinned
    host memory.  Returns (wall seconds, infos)."""
    t0 = time.perf_counter()
    ids = [srv.submit_forward(pin_vol, NPHI, NTHETA, NSHIFT, pin_outs[k % len(pin_outs)],
                              half_extent=HALF_EXTENT, tag=k) for k in range(steps)]
    infos = [srv.wait(i) for i in ids]
    return time.perf_counter() - t0, infos


def serving_mix(wrt, dev, count, seed, budget):
    """A Poisson stream of mixed requests (the serving configuration, scaled to
    `count` requests): edge 64/96/128/192/256 w.p. .30/.25/.20/.15/.10,
    forward (80 %) or adjoint (20 %), sphere grids 32x64 .. 96x192 (latitudes
    x longitudes), 128-384 shifts, FP32 volumes of seeded ellipsoids, seeded
    Gaussian Radon data for the adjoints.  Arrival rate: ~90 % of the measured
    service rate of a first batch."""
    from wrt_b200.phantom import ellipsoid_phantom

    rng = np.random.default_rng(seed)
    edges = rng.choice([64, 96, 128, 192, 256], size=count, p=[0.30, 0.25, 0.20, 0.15, 0.10])
    vol_cache = {}
    reqs = []
    for k in range(count):
        n = int(edges[k])
        nth = int(rng.integers(32, 97))
        ns = int(rng.integers(128, 385))
        if rng.random() < 0.8:
            if n not in vol_cache:
                vol_cache[n] = ellipsoid_phantom(n, 12, seed + n).astype(np.float32)
            reqs.append(("fwd", n, nth, ns))
        else:
            reqs.append(("adj", n, nth, ns))
    adj_data = {}
    with wrt.Server(dev, budget_bytes=budget, max_batch=16, max_inflight=2) as srv:
        def submit(r):
            op, n, nth, ns = r
            if op == "fwd":
                out = np.empty((ns, 2 * nth, nth))
                return srv.submit_forward(vol_cache[n], 2 * nth, nth, ns, out, half_extent=n), out
            key = (nth, ns)
            if key not in adj_data:
                adj_data[key] = rng.standard_normal((ns, 2 * nth, nth))
            out = np.empty((n, n, n))
            return srv.submit_adjoint(adj_data[key], n, out), out
        # service-rate estimate from the first few requests run back to back
        t0 = time.perf_counter()
        warm = [submit(r) for r in reqs[:8]]
        for rid, _ in warm:
            srv.wait(rid)
        rate = 8 / (time.perf_counter() - t0) * 0.9
        gaps = rng.exponential(1.0 / rate, size=count)
        t_start = time.perf_counter()
        pending, t_next = [], t_start
        for k, r in enumerate(reqs):
            t_next += gaps[k]
            delay = t_next - time.perf_counter()
            if delay > 0:
                time.sleep(delay)
            pending.append((r, submit(r)))
        infos = [(r, srv.wait(rid)) for r, (rid, _) in pending]
        wall = time.perf_counter() - t_start
        st = srv.stats()
    lat = np.array([i.done_ms - i.submit_ms for _, i in infos])
    planes = sum(r[3] * 2 * r[2] * r[2] for r, _ in infos if r[0] == "fwd")
    return {"requests": count, "forward": sum(r[0] == "fwd" for r in reqs),
            "arrival_rate_per_s": rate, "wall_s": wall,
            "requests_per_s": count / wall, "plane_integrals_per_s": planes / wall,
            "latency_ms": {"p50": float(np.percentile(lat, 50)),
                           "p99": float(np.percentile(lat, 99))},
            "launches": int(st.launches), "hbm_peak_bytes": int(st.bytes_peak),
            "budget_bytes": int(st.budget),
            "mean_batch": float(np.mean([i.batch_size for _, i in infos]))}


def cli_compare(args):
    """The drop-in programs against the reference's own programs
    (oracle/_ref, compiled from its sources), end to end on the same text
    files, each given all host cores with -n: radon_grid on a 128^3 volume
    file (2,097,152 lines; 32 longitudes x 16 latitudes x 64 shifts, the
    reference's default nearest sampler and 4n x 4n lattice), then
    radon3d_grid of that Radon file back to 64^3.  Wall time per program run
    (start-up, text input, transform, text output), the programs' own
    transform times, and the relative L2 difference of the outputs."""
    import subprocess
    import tempfile

    load_package()
    from wrt_b200.phantom import ellipsoid_phantom

    sys.path.insert(0, str(ROOT))
    import oracle as O

    cores = cpu_threads()
    ours, ref = PKG_DIR / "bin", ROOT / "oracle" / "_ref"
    if not (ref / "radon_grid").exists():
        print(json.dumps({"path": "cli", "unavailable": "oracle/_ref programs not built"}))
        return 0
    n, nphi, ntheta, nshift, n_adj = N, 32, 16, 64, 64
    work = Path(tempfile.mkdtemp(prefix="wrt_cli_"))
    vol = ellipsoid_phantom(n, ELLIPSOIDS, SEED)
    np.savetxt(work / "volume.txt", vol.reshape(-1), fmt="%lf")
    (work / "radon_params.txt").write_text(
        f"{nphi} nphi\n{ntheta} ntheta\n{nshift} nshift\n{n} ngrid\n")
    (work / "adjoint_params.txt").write_text(
        f"{nphi} nphi\n{ntheta} ntheta\n{nshift} nshift\n{n_adj} ngrid\n")
    res = {}
    for who, bindir in (("ours", ours), ("reference", ref)):
        d = work / who
        d.mkdir()
        row = {}
        for prog, params, inp, out in (("radon_grid", "radon_params.txt", "../volume.txt",
                                        "radon.csv"),
                                       ("radon3d_grid", "adjoint_params.txt", "radon.csv",
                                        "adjoint.txt")):
            cmd = [str(bindir / prog), "-p", f"../{params}", "-i", inp, "-o", out, "-n",
                   str(cores)]
            t0 = time.perf_counter()
            r = subprocess.run(cmd, cwd=d, capture_output=True, text=True, timeout=1800)
            wall = time.perf_counter() - t0
            if r.returncode:
                raise RuntimeError(f"{who} {prog} failed: {r.stderr[-500:]}")
            stamp = [ln.strip() for ln in r.stdout.splitlines() if "elapsed" in ln.lower()]
            row[prog] = {"wall_s": wall, "program_reports": stamp}
        res[who] = row
    a = np.loadtxt(work / "ours" / "radon.csv", delimiter=",")[:, 3]
    b = np.loadtxt(work / "reference" / "radon.csv", delimiter=",")[:, 3]
    c = np.loadtxt(work / "ours" / "adjoint.txt")
    d = np.loadtxt(work / "reference" / "adjoint.txt")
    line = {
        "path": "cli", "metric": "drop-in program wall time vs the reference's programs",
        "unit": "s", "higher_is_better": False, "cores": cores,
        "config": {"radon_grid": f"{n}^3 volume text file, {nphi}x{ntheta} directions x {nshift} "
                                 "shifts, nearest sampler, 4n x 4n lattice (the defaults)",
                   "radon3d_grid": f"that Radon file back to {n_adj}^3"},
        "ours": res["ours"], "reference": res["reference"],
        "speedup": {p: res["reference"][p]["wall_s"] / res["ours"][p]["wall_s"]
                    for p in res["ours"]},
        "rel_l2_outputs": {"radon_grid": float(np.linalg.norm(a - b) / np.linalg.norm(b)),
                           "radon3d_grid": float(np.linalg.norm(c - d) / np.linalg.norm(d))},
        "note": "the reference's text values carry 6 decimals (%lf), so the comparison is "
                "limited by the printed precision",
    }
    print(json.dumps(line))
    return 0


def serving_stream(args, dist):
    """The serving configuration at its stated size: `--requests` (10,000)
    transform requests arriving as a seeded Poisson stream, each a volume of
    edge 64/96/128/192/256 (w.p. .30/.25/.20/.15/.10) with a forward Radon
    transform (80 %) or a backprojection of seeded Gaussian Radon data (20 %),
    sphere grids of 32..96 latitudes x twice as many longitudes, 128..384
    shifts, admitted by one wrt_server under a 60 GB HBM budget.  FP32 volumes
    come from 4 seeded ellipsoid phantoms per edge; Radon data are windows of
    one seeded Gaussian pool at seeded offsets.  Arrival rate: 90 % of the
    service rate measured on 32 requests run back to back first.  Reported:
    p50/p99 latency (submission to result in the caller's buffer), requests/s,
    plane integrals/s, lattice samples/s and spline evaluations/s, mean batch,
    launches, peak HBM.  One request in 100 is checked against the FP64 oracle
    on 8 seeded planes (forward) or voxels (backprojection)."""
    import queue

    wrt = load_package()
    from wrt_b200.phantom import ellipsoid_phantom

    sys.path.insert(0, str(ROOT))
    import oracle as O

    count = args.requests
    rng = np.random.default_rng(4000)
    edges = rng.choice([64, 96, 128, 192, 256], size=count, p=[0.30, 0.25, 0.20, 0.15, 0.10])
    nths = rng.integers(32, 97, size=count)
    nss = rng.integers(128, 385, size=count)
    fwd = rng.random(count) < 0.8
    variant = rng.integers(0, 4, size=count)
    pool = rng.standard_normal(16 << 20)
    offsets = rng.integers(0, pool.size - 96 * 96 * 2 * 384, size=count)
    vols = {(n, v): ellipsoid_phantom(n, 12, 5000 + 10 * n + v).astype(np.float32)
            for n in (64, 96, 128, 192, 256) for v in range(4)}

    def make(k):
        n, nth, ns = int(edges[k]), int(nths[k]), int(nss[k])
        if fwd[k]:
            out = np.empty((ns, 2 * nth, nth))
            return ("fwd", n, nth, ns, vols[(n, int(variant[k]))], out)
        size = ns * 2 * nth * nth
        radon = pool[offsets[k]:offsets[k] + size].reshape(ns, 2 * nth, nth)
        return ("adj", n, nth, ns, radon, np.empty((n, n, n)))

    def submit(srv, r, tag):
        op, n, nth, ns, data, out = r
        if op == "fwd":
            return srv.submit_forward(data, 2 * nth, nth, ns, out, half_extent=n, tag=tag)
        return srv.submit_adjoint(data, n, out, tag=tag)

    checks = []
    with wrt.Server(0, budget_bytes=60 << 30, max_batch=16, max_inflight=2) as srv:
        # service rate: 32 requests of the same distribution back to back
        warm = [make(k) for k in range(32)]
        t0 = time.perf_counter()
        ids = [submit(srv, r, 0) for r in warm]
        for i in ids:
            srv.wait(i)
        service = 32 / (time.perf_counter() - t0)
        rate = 0.9 * service
        gaps = np.random.default_rng(4001).exponential(1.0 / rate, size=count)
        done = queue.Queue()
        infos = [None] * count

        def waiter():
            while True:
                item = done.get()
                if item is None:
                    return
                k, rid, r = item
                infos[k] = srv.wait(rid)
                if k % 100 == 0:
                    checks.append((k, r))
        th = threading.Thread(target=waiter, daemon=True)
        th.start()
        clocks = ClockSampler(0)
        clocks.start()
        t_start = time.perf_counter()
        t_next = t_start
        for k in range(count):
            t_next += gaps[k]
            delay = t_next - time.perf_counter()
            if delay > 0:
                time.sleep(delay)
            r = make(k)
            done.put((k, submit(srv, r, k), r))
        done.put(None)
        th.join()
        wall = time.perf_counter() - t_start
        clk = clocks.stop()
        st = srv.stats()
    lat = np.array([i.done_ms - i.submit_ms for i in infos])
    queue_ms = np.array([i.start_ms - i.submit_ms for i in infos])
    planes = int(sum(int(nss[k]) * 2 * int(nths[k]) ** 2 for k in range(count) if fwd[k]))
    lattice = int(sum(int(nss[k]) * 2 * int(nths[k]) ** 2 * (2 * int(edges[k])) ** 2
                      for k in range(count) if fwd[k]))
    evals = int(sum(int(edges[k]) ** 3 * 2 * int(nths[k]) ** 2 for k in range(count) if not fwd[k]))
    # oracle spot checks of the served results
    errs = []
    crng = np.random.default_rng(4002)
    for k, (op, n, nth, ns, data, out) in sorted(checks, key=lambda c: c[0]):
        if op == "fwd":
            phi, theta, _, shift = O.radon_grid(2 * nth, nth, ns)
            sel = crng.integers(0, [ns, 2 * nth, nth], size=(8, 3))
            ref = O.radon_planes(data, phi[sel[:, 1]], theta[sel[:, 2]], shift[sel[:, 0]],
                                 sampler=O.TRILINEAR, half_extent=n)
            got = out[sel[:, 0], sel[:, 1], sel[:, 2]]
        else:
            sel = crng.integers(0, n, size=(8, 3))  # iz, ix, iy
            c = lambda i: -1.0 + (2.0 * i + 1.0) / n
            ref = O.adjoint_points(data, c(sel[:, 1]), c(sel[:, 2]), c(sel[:, 0]))
            got = out[sel[:, 0], sel[:, 1], sel[:, 2]]
        den, dif = float(np.linalg.norm(ref)), float(np.linalg.norm(got - ref))
        # planes all outside the volume's support: exactly 0 on both sides
        rel = dif / den if den > 0 else (0.0 if dif == 0 else float("inf"))
        errs.append({"request": k, "op": op, "n": n, "grid": [nth, 2 * nth, ns], "rel_l2": rel,
                     "exact_zero": den == 0 and dif == 0})
    worst = max(e["rel_l2"] for e in errs)
    print(json.dumps({
        "metric": "served requests/s, 10,000-request Poisson stream (p50/p99 ms)",
        "value": count / wall, "unit": "requests/s", "n_gpus": 1, "higher_is_better": True,
        "path": "serving", "dtype": "f32", "data": "synthetic",
        "config": {"workload": "serving: Poisson arrivals, edge 64/96/128/192/256 w.p. "
                               ".30/.25/.20/.15/.10, 80/20 forward/adjoint, grids 32x64..96x192, "
                               "128-384 shifts, FP32 volumes, 60 GB HBM budget",
                   "requests": count, "max_batch": 16, "max_inflight": 2},
        "requests": count, "completed": int(st.completed), "failed": int(st.failed),
        "forward": int(fwd.sum()), "adjoint": int(count - fwd.sum()),
        "service_rate_per_s": service, "arrival_rate_per_s": rate, "wall_s": wall,
        "latency_ms": {"p50": float(np.percentile(lat, 50)), "p90": float(np.percentile(lat, 90)),
                       "p99": float(np.percentile(lat, 99)), "max": float(lat.max())},
        "queue_ms": {"p50": float(np.percentile(queue_ms, 50)),
                     "p99": float(np.percentile(queue_ms, 99))},
        "plane_integrals_per_s": planes / wall, "lattice_samples_per_s": lattice / wall,
        "spline_evaluations_per_s": evals / wall,
        "samples_definition": "forward: (2n)^2 lattice points per plane (the benchmark lattice, "
                              "before cropping); adjoint: n^3 x directions spline evaluations",
        "mean_batch": float(np.mean([i.batch_size for i in infos])),
        "launches": int(st.launches), "hbm_peak_bytes": int(st.bytes_peak),
        "budget_bytes": int(st.budget), "clocks": clk,
        "oracle_checks": {"requests_checked": len(errs), "per_request": "8 seeded planes or voxels",
                          "max_rel_l2": worst, "tolerance": 1e-5, "all_within": worst <= 1e-5,
                          "median_rel_l2": float(np.median([e["rel_l2"] for e in errs])),
                          "worst": sorted(errs, key=lambda e: -e["rel_l2"])[:3]}}))
    return 0


def run_ours(args, dist):
    wrt = load_package()
    from wrt_b200.phantom import ellipsoid_phantom

    dev = dist.local_rank
    ctx = wrt.Context(dev)
    phantom = ellipsoid_phantom(N, ELLIPSOIDS, SEED)
    vol = wrt.Volume(ctx, N)
    vol.upload(phantom.astype(np.float32))
    grid = wrt.Grid(ctx, NPHI, NTHETA, NSHIFT)
    nplanes = grid.nplanes
    out = wrt.DeviceBuffer(ctx, nplanes * 8)
    kernel = {"plain": wrt.KERNEL_PLAIN, "staged": wrt.KERNEL_STAGED,
              "auto": wrt.KERNEL_AUTO}[args.kernel]

    def step(k=kernel):
        if k == wrt.KERNEL_PLAIN:
            wrt.radon_forward_device(ctx, vol, grid, out.ptr, sampler=wrt.TRILINEAR,
                                     half_extent=HALF_EXTENT, kernel=k)
        else:  # the batched persistent kernel through its captured graph
            wrt.radon_forward_batch(ctx, [(vol, grid, out.ptr, HALF_EXTENT)])

    # the autotuner picks the staged kernel's tile shape on this request
    tile = None
    if kernel != wrt.KERNEL_PLAIN:
        if args.tile is not None:
            best, best_ms = args.tile, None
            wrt.set_plane_kernel_config(ctx, best)
        else:
            best, best_ms = wrt.tune_plane_kernel(ctx, vol, grid, out.ptr, sampler=wrt.TRILINEAR,
                                                  half_extent=HALF_EXTENT)
        t, g, s = wrt.plane_kernel_configs()[best]
        tile = {"threads": t, "rows_per_warp_group": g, "shifts_per_lane": s,
                "tuner_ms": best_ms}

    # samples evaluated per launch (one counted launch, outside the timed region)
    ctx.count_samples(True)
    step()
    samples = ctx.sample_count()
    ctx.count_samples(False)

    for _ in range(max(args.warmup, 3)):
        step()
    ctx.synchronize()

    clocks = ClockSampler(dev)
    clocks.start()
    dist.barrier()
    ctx.synchronize()
    launches0 = ctx.launches
    times = []
    for _ in range(args.steps):
        ctx.flush_l2()
        ctx.timer_start()
        step()
        times.append(ctx.timer_stop())
    launches = ctx.launches - launches0
    ctx.synchronize()
    dist.barrier()
    clk = clocks.stop()
    total_ms = dist.max(sum(times))
    ms_per_step = total_ms / args.steps
    value = nplanes * args.steps * dist.world / (total_ms * 1e-3)
    result_dev = out.download(np.empty((NSHIFT, NPHI, NTHETA)))

    if args.only_kernel:  # profiling captures: the timed kernel launches and nothing else
        if dist.rank == 0:
            print(json.dumps({"metric": METRIC, "value": value, "unit": UNIT,
                              "ms_per_step": ms_per_step, "samples_per_step": samples,
                              "tile": tile, "note": "kernel only (profiling run)"}))
        out.close(); vol.close(); grid.close(); ctx.close()
        return 0

    # plain kernel alongside (the one-request-per-launch baseline)
    plain = None
    if kernel != wrt.KERNEL_PLAIN:
        step(wrt.KERNEL_PLAIN)
        pt = []
        for _ in range(max(2, min(args.steps, 5))):
            ctx.flush_l2()
            ctx.timer_start()
            step(wrt.KERNEL_PLAIN)
            pt.append(ctx.timer_stop())
        plain_res = out.download(np.empty((NSHIFT, NPHI, NTHETA)))
        plain = {"value": nplanes / (statistics.mean(pt) * 1e-3), "unit": UNIT,
                 "ms_per_step": statistics.mean(pt),
                 "rel_l2_vs_staged": float(np.linalg.norm(plain_res - result_dev) /
                                           np.linalg.norm(result_dev))}

    # end to end through the serving loop (the public API a caller uses): each
    # step is one request of the workload, its FP32 volume copied in from pinned
    # host memory and its FP64 plane integrals copied back to pinned host memory
    pin_vol = wrt.PinnedArray(ctx, (N, N, N), np.float32)
    pin_vol.array[...] = phantom
    pin_outs = [wrt.PinnedArray(ctx, (NSHIFT, NPHI, NTHETA), np.float64) for _ in range(4)]
    srv = wrt.Server(dev, budget_bytes=4 << 30, max_batch=8, max_inflight=2)
    served_stream(wrt, srv, pin_vol.array, [p.array for p in pin_outs], 3)  # warm-up
    dist.barrier()
    wall, infos = served_stream(wrt, srv, pin_vol.array, [p.array for p in pin_outs], args.steps)
    served_res = np.array(pin_outs[(args.steps - 1) % len(pin_outs)].array)
    srv.close()
    wall = dist.max(wall)
    e2e_value = nplanes * args.steps * dist.world / wall
    lat = np.array([i.done_ms - i.submit_ms for i in infos])
    served_equal = bool(np.array_equal(served_res, result_dev))

    # compulsory HBM bytes, and the lattice's samples at 32 B each against the
    # measured shared-memory bandwidth of this device
    smem_bw = ctx.smem_bandwidth()
    per_launch_s = ms_per_step * 1e-3
    achieved = samples * BYTES_PER_SAMPLE / per_launch_s / 1e9
    peak = smem_bw / 1e9
    hbm_bytes = N ** 3 * 4 + nplanes * 8  # compulsory: FP32 volume in, FP64 results out
    peaks_file = ROOT / "MEASURED_PEAKS.json"
    hbm_peak = json.loads(peaks_file.read_text()).get("hbm_gbs") if peaks_file.exists() else 6650.0

    result = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": dist.world,
        "steps": args.steps, "warmup": max(args.warmup, 3), "ms_per_step": ms_per_step,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic",
        "config": {"workload": "radon_grid forward, 128^3 volume of 16 seeded ellipsoids, "
                               "64x128 Gauss-uniform sphere grid x 256 shifts, trilinear, "
                               "lattice step 1/n on [-n,n)^2",
                   "n": N, "sphere_grid": [NTHETA, NPHI], "shifts": NSHIFT,
                   "planes_per_step": nplanes, "kernel": args.kernel, "tile": tile,
                   "path": "batch entry point (wrt_radon_forward_batch): row-sum profiles",
                   "l2": "flushed before every timed step (2x L2 memset)",
                   "parallelism": f"replicas x{dist.world}"},
        "samples_per_step": samples,
        "samples_per_s": samples * args.steps * dist.world / (total_ms * 1e-3),
        "gpu_launches": launches,
        "roofline": {"bound": "latency", "achieved": hbm_bytes / per_launch_s / 1e9,
                     "peak": hbm_peak, "unit": "GB/s",
                     "frac": hbm_bytes / per_launch_s / 1e9 / hbm_peak,
                     "note": "compulsory HBM bytes (volume in, results out); the kernel reads its "
                             "row sums from tables in L2 and waits for those gathers",
                     "lattice": {"achieved": achieved, "peak": peak, "unit": "GB/s",
                                 "note": "32 B per trilinear sample of the lattice against the "
                                         "shared-memory read bandwidth measured in this run "
                                         "(wrt_measure_smem_bandwidth): what evaluating every "
                                         "sample would have to read.  The samples of a row share "
                                         "its table entry, so this may exceed the peak"}},
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": N ** 3 * 4,
                "d2h_bytes_per_step": nplanes * 8,
                "path": "wrt_server: one request per step, pinned FP32 volume in, pinned FP64 "
                        "results out, 2 launches in flight",
                "latency_ms": {"p50": float(np.percentile(lat, 50)),
                               "p99": float(np.percentile(lat, 99))},
                "result_bitwise_equal_to_kernel_path": served_equal},
        "clocks": clk,
    }
    if plain:
        result["plain"] = plain
        result["served_over_plain"] = e2e_value / plain["value"]
    if not args.no_other_paths:
        result["paths"] = other_paths(wrt, ctx, phantom, max(3, min(args.steps, 10)), args.warmup,
                                      smem_bw, hbm_peak, dist.rank == 0 and not args.no_cpu_baseline)
        result["batch_vs_one_per_launch"] = batch_vs_one_per_launch(wrt, ctx, 3)
        result["batch_vs_one_per_launch_small"] = batch_vs_one_per_launch(
            wrt, ctx, 3, count=256, edges=(16, 24, 32, 48), lat=(8, 17), shifts=(32, 65),
            seed=2003)
        result["configs"] = config_runs(wrt, ctx, 2)
    if dist.rank == 0 and dist.world == 1 and not args.no_serving_mix:
        result["serving"] = serving_mix(wrt, dev, args.mix_requests, 4000, 60 << 30)
    if dist.rank == 0 and dist.world == 1 and not args.no_cpu_baseline:
        result["cpu_baseline"] = cpu_baseline(phantom)
    if dist.rank == 0:
        print(json.dumps(result))
    pin_vol.close()
    for p in pin_outs:
        p.close()
    out.close()
    vol.close()
    grid.close()
    ctx.close()
    return 0


# ------------------------------------------------------------ other paths
PATHS = {
    # path: (metric, unit, workload)
    "ray": ("rays/s @128^3 (128 layers x 128 shifts x 128 angles, reference frame)", "rays/s",
            "ray_grid, 128^3 volume of 16 seeded ellipsoids, 128 z-layers x 128 shifts x 128 "
            "angles, trilinear, 513 samples per ray (255 inside the unit ball)"),
    "ray_rotated": ("rays/s @128^3 (128 layers x 128 shifts x 128 angles, rotated frame)",
                    "rays/s",
                    "ray_grid in one seeded random rotation of the layer frame (one of the "
                    "configuration's orientations), 128^3 volume, 128 layers x 128 shifts x 128 "
                    "angles, trilinear"),
    "reduction": ("plane integrals/s from 128^3 ray data (64x128 sphere grid x 256 shifts)",
                  "plane integrals/s",
                  "radon_reduction, rays 128 layers x 128 shifts x 128 angles -> 64x128 sphere "
                  "grid x 256 shifts (ray shift grid decoupled: spline over 128 offsets)"),
    "nearest": ("plane integrals/s @128^3 (64x128 sphere grid x 256 shifts, nearest sampler, "
                "512^2 lattice)", "plane integrals/s",
                "radon_grid with the reference's defaults: zero_interp, lattice [-2n, 2n)^2 with "
                "step 1/n, 128^3 volume of 16 seeded ellipsoids, 64x128 sphere grid x 256 shifts"),
    "adjoint": ("voxels/s of the backprojection to 128^3 (64x128 sphere grid x 256 shifts)",
                "voxels/s",
                "radon3d_adjoint, seeded N(0,1) Radon data 64x128 sphere grid x 256 shifts -> "
                "128^3 voxels, 8192 spline evaluations per voxel"),
}


def run_path(args, dist):
    """One of the other hot paths through its drop-in entry point (host arrays
    in and out, as the reference's programs take them): K timed calls after W
    warm-up calls, CUDA events on the library's stream around each call (the
    calls are synchronous, so this is end to end), the reference's own code on
    a bounded sample of the same workload on the host cores beside it."""
    wrt = load_package()
    from wrt_b200.phantom import ellipsoid_phantom

    sys.path.insert(0, str(ROOT))
    import oracle as O

    metric, unit, workload = PATHS[args.path]
    ctx = wrt.Context(dist.local_rank)
    n = N
    rng = np.random.default_rng(SEED)
    vol = ellipsoid_phantom(n, ELLIPSOIDS, SEED)
    frame = None
    if args.path == "ray_rotated":
        q, r = np.linalg.qr(rng.standard_normal((3, 3)))
        frame = q * np.sign(np.diag(r))
        if np.linalg.det(frame) < 0:
            frame[:, 0] = -frame[:, 0]
    if args.path in ("ray", "ray_rotated"):
        call = lambda: ctx.ray_grid(vol, n, 128, 128, frame=frame)
        units, h2d, d2h = n * 128 * 128, vol.nbytes, n * 128 * 128 * 8
    elif args.path == "reduction":
        rays = ctx.ray_grid(vol, n, 128, 128)
        call = lambda: ctx.radon_reduction(rays, NSHIFT, NTHETA)
        units, h2d, d2h = NSHIFT * NPHI * NTHETA, rays.nbytes, NSHIFT * NPHI * NTHETA * 8
    elif args.path == "nearest":
        call = lambda: ctx.radon_grid(vol, NPHI, NTHETA, NSHIFT, sampler=wrt.NEAREST)
        units, h2d, d2h = NSHIFT * NPHI * NTHETA, vol.nbytes, NSHIFT * NPHI * NTHETA * 8
    else:
        radon = rng.standard_normal((NSHIFT, NPHI, NTHETA))
        call = lambda: ctx.radon3d_adjoint(radon, n)
        units, h2d, d2h = n ** 3, radon.nbytes, n ** 3 * 8
    for _ in range(max(args.warmup, 3)):
        result = call()
    ctx.synchronize()
    clocks = ClockSampler(dist.local_rank)
    clocks.start()
    dist.barrier()
    times = []
    for _ in range(args.steps):
        ctx.timer_start()
        result = call()
        times.append(ctx.timer_stop())
    dist.barrier()
    clk = clocks.stop()
    total_ms = dist.max(sum(times))
    value = units * args.steps * dist.world / (total_ms * 1e-3)

    # the reference on the host cores: a bounded seeded sample of the same units
    cpu = None
    if dist.rank == 0 and not args.no_cpu_baseline and O.Reference.available():
        ref, cores = O.Reference(), cpu_threads()
        t0 = time.perf_counter()
        if args.path == "ray":
            m = 65536
            idx = rng.integers(0, units, size=m)
            s_grid, phi_grid = O.ray_grid(128, 128)
            z = -1.0 + (idx // (128 * 128)) * (2.0 / (n - 1))
            got = ref.rays(vol, z, s_grid[(idx // 128) % 128], phi_grid[idx % 128], cores)
            ours = result.reshape(-1)[idx]
        elif args.path == "ray_rotated":
            # the reference has no layer frames: the FP64 restatement, all rays
            m = units
            got = O.ray_forward(vol, n, 128, 128, frame=frame, nthreads=cores).reshape(-1)
            ours = result.reshape(-1)
        elif args.path == "nearest":
            m = 1024
            idx = rng.integers(0, units, size=m)
            phi, theta, _, shift = O.radon_grid(NPHI, NTHETA, NSHIFT)
            got = ref.plane_integrals(vol, phi[(idx // NTHETA) % NPHI], theta[idx % NTHETA],
                                      shift[idx // (NPHI * NTHETA)], cores)
            ours = result.reshape(-1)[idx]
        elif args.path == "reduction":
            m = 4096
            idx = rng.integers(0, units, size=m)
            # the reference couples the ray and Radon shift grids: rays on 256 shifts
            rays_c = ctx.ray_grid(vol, n, NSHIFT, 128)
            t0 = time.perf_counter()
            got = ref.reduction_planes(rays_c, NTHETA, idx // (NPHI * NTHETA),
                                       (idx // NTHETA) % NPHI, idx % NTHETA, cores)
            ours = None
        else:
            m = 64
            idx = rng.integers(0, units, size=m)
            iz, ix, iy = idx // (n * n), (idx // n) % n, idx % n
            c = lambda i: -1.0 + (2.0 * i + 1.0) / n
            got = ref.adjoint_points(radon, c(ix), c(iy), c(iz), cores)
            ours = result.reshape(-1)[idx]
        wall = time.perf_counter() - t0
        cpu = {"value": m / wall, "unit": unit, "cores": cores, "kind": "reference",
               "sample": f"{m} seeded random units of this workload, the reference's own code "
                         "(oracle/_ref) with OpenMP over units"}
        if args.path == "ray_rotated":
            cpu.update(kind="port", sample=f"all {m} rays, the FP64 oracle restatement with the "
                                           "frame (the reference has no layer frames)")
        if ours is not None:
            cpu["rel_l2_gpu_vs_reference_on_sample"] = float(
                np.linalg.norm(ours - got) / max(np.linalg.norm(got), 1e-300))
    if dist.rank == 0:
        print(json.dumps({
            "metric": metric, "value": value, "unit": unit, "n_gpus": dist.world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": total_ms / args.steps,
            "ms_per_step_median": statistics.median(times),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "path": args.path,
            "config": {"workload": workload, "api": "drop-in entry point, host arrays"},
            "e2e": {"value": value, "unit": unit, "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h},
            "clocks": clk, "cpu_baseline": cpu}))
    ctx.close()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--kernel", choices=["auto", "plain", "staged"], default="auto")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-serving-mix", action="store_true")
    ap.add_argument("--no-other-paths", action="store_true",
                    help="skip the ray / reduction / adjoint and batching measurements")
    ap.add_argument("--only-kernel", action="store_true",
                    help="time the kernel steps only (for profiling captures)")
    ap.add_argument("--mix-requests", type=int, default=96,
                    help="requests in the mixed serving stream")
    ap.add_argument("--tile", type=int, default=None,
                    help="use this tile configuration of the staged kernel instead of tuning")
    ap.add_argument("--requests", type=int, default=10000,
                    help="--path serving: requests in the Poisson stream")
    ap.add_argument("--path", choices=["forward", "serving", "cli", *PATHS], default="forward",
                    help="forward: the headline (plane integrals at 128^3); ray, reduction, "
                         "adjoint: the other hot paths through their drop-in entry points")
    ap.add_argument("--grid", default=None,
                    help="NPHI,NTHETA,NSHIFT: a smaller sphere grid (profiling captures only)")
    args = ap.parse_args()
    if args.grid:
        global NPHI, NTHETA, NSHIFT
        NPHI, NTHETA, NSHIFT = (int(x) for x in args.grid.split(","))
    dist = Dist(args.gpus)
    try:
        if args.path == "serving":
            rc = serving_stream(args, dist) if args.impl == "ours" and dist.rank == 0 else 0
        elif args.path == "cli":
            rc = cli_compare(args) if args.impl == "ours" and dist.rank == 0 else 0
        elif args.path != "forward":
            rc = run_path(args, dist) if args.impl == "ours" else 0
        else:
            rc = run_reference(args, dist) if args.impl == "reference" else run_ours(args, dist)
    finally:
        dist.close()
    return rc


if __name__ == "__main__":
    sys.exit(main())
