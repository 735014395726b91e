"""Benchmark of the MoM impedance-matrix assembly (triangle pairs per second).

Workload (default ``mom_ref_L5``): icosphere level 5 -- 20480 triangles, 10242 vertices,
30720 RWG unknowns -- radius 1 m, ka = 10 (k = 10), the reference's formulation and rule
(EFIE + MFIE summed, collapsed Gauss-Legendre gaussQR = 4: 16 test x 9 source points per
face-edge entry, rotated per local edge, i.e. 1296 kernel evaluations per triangle pair),
float32 arithmetic, Z accumulated straight into the [E, E] complex64 RWG matrix (7.55 GB).
A step zeroes Z and assembles all F^2 triangle pairs.  Synthetic mesh (the reference's
mesh assets are not shipped); the output (7.55 GB) is larger than L2 and is rewritten
every step, so no stale lines survive between steps.

``python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]``
prints one JSON line (rank 0).  Under torchrun each rank assembles its own replica (the
path has no exchange step: replicas only) and the slowest rank's time is reported.

``--impl reference`` times the reference's own algorithm on the host cores instead: the
host build of its CUDA kernel bodies where that exists (oracle/_ref), else the CPU
restatement in oracle/ (float32 build), on a bounded sample of face-edge rows.
"""
from __future__ import annotations

import argparse
import importlib
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, REPO)

WORKLOADS = {
    # name: (icosphere level, k, gaussQR of the reference rule, or 0 for the 7-point EFIE)
    "mom_ref_L5": (5, 10.0, 4),
    "mom_ref_L4": (4, 6.0, 4),
    "mom_ref_L3": (3, 2.0, 4),
    "mom_sym_L5": (5, 10.0, 0),
    "mom_sym_L4": (4, 6.0, 0),
    # ray queries: (terrain cells per side, icospheres, cameras); 512 x 256 skydome rays each
    "ray_skydome": (512, 12, 8),
    # Laplace single-layer collocation, unit Dirichlet data on the sphere: (level, radius, dtype)
    "laplace_col_L5": (5, 1.0, "f32"),
    "laplace_col_L5_f64": (5, 1.0, "f64"),
    # many incidences on one mesh: (ellipsoid level, k, Fibonacci directions x 2 polarisations)
    "mrhs_ell4": (4, 6.0, 256),
    "mrhs_ell4_efie": (4, 6.0, 256),
    # the tensor-core product alone: (unknowns E, right-hand sides m)
    "cgemm_E7680_m512": (7680, 512, 0),
    # uneven meshes in one batch: (meshes, incidences per mesh, seed)
    "batch_star64": (64, 4, 0),
    "batch_star64_efie": (64, 4, 0),
    "batch_star8": (8, 4, 0),
    "batch_star8_efie": (8, 4, 0),
    # scattered H on a field-point grid from vertex currents: (icosphere level, k, grid points per side)
    "radiate_L5": (5, 10.0, 1024),
    # GPU mesh topology (unique edges + face-edge map + edge faces, near-pair list, Z-row map)
    "topology_L7": (7,),
    # the reference's own Laplace path (demo_Laplace_3d.py): Dirichlet solve with its rule, P1:
    # (icosphere level, gaussQR, radius)
    "laplace_ref_L4": (4, 2, 0.5),
    # its operator assembly alone: V and K panels [F, F, 3, 3] with the same rule and relation
    "laplace_panels_L4": (4, 2, 0.5),
    "laplace_panels_L5": (5, 2, 0.5),
    # the ferrofluid pressure projection (MeshPressure.solve), hydrostatic droplet: (icosphere level,)
    "pressure_L4": (4,),
    # Laplace mixed Dirichlet / Neumann solve, u = z on the unit sphere: (icosphere level, dtype)
    "laplace_mixed_L4": (4, "f32"),
    "laplace_mixed_L3": (3, "f32"),
    # the mixed-precision EFIE solve alone (assembly + SAI + half copy + preconditioned GMRES to
    # a 3e-5 residual, i.e. a <1e-4 error in J): (icosphere level, k)
    "efie_solve_L5": (5, 10.0),
    "efie_solve_L4": (4, 10.0),
    # learned initial guess: (training meshes, held-out meshes, incidences per mesh)
    "learned_star": (5000, 256, 4),
    "learned_star_small": (500, 64, 4),
}


def _args():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=5)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--workload", choices=sorted(WORKLOADS), default="mom_ref_L5")
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-solve", action="store_true",
                   help="skip the GMRES time-to-solution report after the timed region")
    p.add_argument("--cpu-seconds", type=float, default=10.0,
                   help="target CPU work per reference-arm / baseline sample")
    return p.parse_args()


# ---------------------------------------------------------------------------------------
# clocks sampled during the timed region
# ---------------------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.samples = []
        self._proc = None
        self._thread = None

    def start(self):
        try:
            self._proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except (FileNotFoundError, OSError):
            self._proc = None
            return
        self._thread = threading.Thread(target=self._read, daemon=True)
        self._thread.start()

    def _read(self):
        for line in self._proc.stdout:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 8:
                self.samples.append(parts)

    def stop(self):
        if self._proc is not None:
            self._proc.terminate()
            try:
                self._proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self._proc.kill()
        if self._thread is not None:
            self._thread.join(timeout=5)

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"], "samples": 0}
        sm = [float(s[0]) for s in self.samples if s[0].replace(".", "").isdigit()]
        smax = [float(s[1]) for s in self.samples if s[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for s in self.samples:
            for i, n in enumerate(names):
                if s[4 + i].lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(self.samples)}


# ---------------------------------------------------------------------------------------
# replicas: one process per GPU, each timing its own copy of the workload (no exchange step)
# ---------------------------------------------------------------------------------------
def replica_barrier(world, dev=None):
    """All ranks meet (torch.distributed.barrier when world > 1); then the device idles."""
    import torch

    if world > 1:
        torch.distributed.barrier()
    if dev is not None and dev.type == "cuda":
        torch.cuda.synchronize(dev)


def replica_max(value, world, dev=None):
    """The largest of every rank's value (the slowest replica's time) -- all ranks get it."""
    if world <= 1:
        return float(value)
    import torch

    t = torch.tensor([float(value)], dtype=torch.float64, device=dev if dev is not None else "cpu")
    torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    return float(t.item())


# ---------------------------------------------------------------------------------------
# CPU reference / baseline
# ---------------------------------------------------------------------------------------
def _mesh_np(level):
    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    v, f = pkg.meshes.icosphere(level)
    v32 = v.astype(np.float32)
    p0, p1, p2 = (v32[f[:, i]].astype(np.float32) for i in range(3))
    cr = np.cross(p1 - p0, p2 - p1)
    areas = (0.5 * np.linalg.norm(cr, axis=1)).astype(np.float32)
    normals = (cr / np.linalg.norm(cr, axis=1, keepdims=True)).astype(np.float32)
    return v32, f, areas, normals


def _rules_np(gq):
    def gl(n):
        x, w = np.polynomial.legendre.leggauss(n)
        x = x.astype(np.float32)
        w = w.astype(np.float32)
        return (x + np.float32(1)) / np.float32(2), w / np.float32(2)
    px, wx = gl(gq)
    py, wy = gl(gq - 1)
    return px, wx, py, wy


def cpu_sample_run(workload, seconds, steps=1, warmup=0):
    """Time the reference algorithm on host cores over a bounded sample of face-edge rows.

    Runs the C restatement of the reference kernel (oracle/, float32 build, one OpenMP
    thread per host core).  The host build of the reference's own kernel bodies
    (oracle/_ref) is not used for timing: its 32-bit flat index overflows beyond
    F = 15447 faces (mesh_MOM_3d.cu:364-374) and it has no row window.  Returns
    (pairs_per_s list, info dict).
    """
    from oracle import oracle as O

    level, k, gq = WORKLOADS[workload]
    v, f, a, n = _mesh_np(level)
    px, wx, py, wy = _rules_np(gq)
    nf = f.shape[0]
    threads = os.cpu_count() or 1
    os.environ.setdefault("OMP_NUM_THREADS", str(threads))

    def run(rows):
        t0 = time.perf_counter()
        O.mom_zmat_fe(v, f, a, n, px, wx, py, wy, k, rows=(0, rows), dtype=np.float32)
        return time.perf_counter() - t0

    calib_rows = 6
    t = run(calib_rows)
    rate_rows = calib_rows / max(t, 1e-6)
    rows = max(3, min(3 * nf, int(rate_rows * seconds)))
    for _ in range(warmup):
        run(max(3, rows // 4))
    vals, step_ms = [], []
    for _ in range(steps):
        dt = run(rows)
        vals.append(rows * 3 * nf / 9.0 / dt)  # face-edge entries / 9 = triangle pairs
        step_ms.append(dt * 1e3)
    info = {"kind": "port", "cores": threads,
            "sample": f"{rows} of {3 * nf} face-edge test rows x all {3 * nf} columns "
                      f"({rows * nf // 3} triangle-pair equivalents), float32 C restatement",
            "sample_ms_per_step": statistics.mean(step_ms)}
    return vals, info


# ---------------------------------------------------------------------------------------
# ray-query workload
# ---------------------------------------------------------------------------------------
def ray_scene(cells, n_spheres, seed=0):
    """Height-field terrain (2 cells^2 faces) on [-50, 50]^2 plus icospheres (L5) above it."""
    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    xs = np.linspace(-50.0, 50.0, cells + 1)
    X, Y = np.meshgrid(xs, xs, indexing="ij")
    Z = 2.0 * np.sin(0.11 * X) * np.cos(0.07 * Y) + 0.5 * np.sin(0.5 * X + 0.3 * Y)
    verts = [np.stack([X, Y, Z], -1).reshape(-1, 3)]
    i, j = np.meshgrid(np.arange(cells), np.arange(cells), indexing="ij")
    a = (i * (cells + 1) + j).ravel()
    b, c, d = a + cells + 1, a + 1, a + cells + 2
    faces = [np.stack([np.stack([a, b, c], -1), np.stack([b, d, c], -1)], 1).reshape(-1, 3)]
    sv, sf = pkg.meshes.icosphere(5, 1.0)
    rng = np.random.default_rng(seed)
    off = verts[0].shape[0]
    for _ in range(n_spheres):
        r = rng.uniform(1.0, 4.0)
        ctr = np.array([rng.uniform(-40, 40), rng.uniform(-40, 40), rng.uniform(4.0, 12.0)])
        verts.append(sv * r + ctr)
        faces.append(sf + off)
        off += sv.shape[0]
    return np.concatenate(verts).astype(np.float32), np.concatenate(faces).astype(np.int32)


def skydome_dirs(n_theta):
    th = (np.arange(n_theta) + 0.5) * np.pi / n_theta
    ph = (np.arange(2 * n_theta) + 0.5) * np.pi / n_theta
    T, P = np.meshgrid(th, ph, indexing="ij")
    return np.stack([np.sin(T) * np.cos(P), np.sin(T) * np.sin(P), np.cos(T)], -1).reshape(-1, 3)


def ray_cameras(n, seed=1):
    rng = np.random.default_rng(seed)
    return np.stack([rng.uniform(-30, 30, n), rng.uniform(-30, 30, n), rng.uniform(3.0, 15.0, n)], 1)


def main_rays(args, rank, world, local_rank):
    cells, n_spheres, n_cam = WORKLOADS[args.workload]
    n_theta = 256
    n_rays = 2 * n_theta * n_theta
    config = {"workload": args.workload, "scene": f"height-field terrain {cells}x{cells} cells + "
              f"{n_spheres} icospheres L5", "cameras": n_cam, "rays_per_camera": n_rays,
              "image": f"{2 * n_theta}x{n_theta} skydome (equirectangular)", "tmin": 0.001, "tmax": 10000.0,
              "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference's ray query is a Vulkan "
                              "ray-tracing pipeline; no graphics stack: unavailable on this box"}), flush=True)
        return
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl")
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    v_np, f_np = ray_scene(cells, n_spheres)
    config["n_faces"] = int(f_np.shape[0])
    verts = torch.from_numpy(v_np).to(dev)
    faces = torch.from_numpy(f_np).to(dev)
    stream = torch.cuda.current_stream(dev)
    b0, b1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    b0.record(stream)
    app = pkg.ray_query.RayQueryApp(verts, faces, device=dev)
    b1.record(stream)
    torch.cuda.synchronize(dev)
    build_ms = b0.elapsed_time(b1)
    cams_np = ray_cameras(n_cam).astype(np.float32)
    dirs_np = np.broadcast_to(skydome_dirs(n_theta), (n_cam, n_rays, 3)).astype(np.float32)
    origins = torch.from_numpy(cams_np).to(dev)
    dirs = torch.from_numpy(np.ascontiguousarray(dirs_np)).to(dev)
    out = torch.empty(n_cam, n_rays, 4, dtype=torch.float32, device=dev)
    total_rays = n_cam * n_rays

    def barrier():
        if world > 1:
            torch.distributed.barrier()
        torch.cuda.synchronize(dev)

    for _ in range(args.warmup):
        app.query(origins, dirs, out=out)
    barrier()
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    # inputs (12.6 MB) + output (16.8 MB) fit in L2; the BVH (~50 MB) too: steady-state
    # numbers for repeated queries of one scene, as a renderer issues them
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    barrier()
    for e0, e1 in ev:
        e0.record(stream)
        app.query(origins, dirs, out=out)
        e1.record(stream)
    barrier()
    clocks.stop()
    ms = [a.elapsed_time(b) for a, b in ev]
    total_ms = sum(ms)
    if world > 1:
        t = torch.tensor([total_ms], device=dev)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        total_ms = float(t.item())
    ms_per_step = total_ms / args.steps
    value = world * total_rays / (ms_per_step / 1e3)
    hit_frac = float((out[..., 0] >= 0).float().mean())
    peaks = pkg.roofline.measured_peaks(REPO)
    hbm = float(peaks.get("hbm_gbs", 6800.0))
    stream_bytes = total_rays * (12 + 16) + n_cam * 12
    ach = stream_bytes / (ms_per_step / 1e3) / 1e9
    line = {"metric": "closest-hit rays/s", "value": value, "unit": "rays/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic", "config": config,
            "roofline": {"bound": "hbm", "achieved": ach, "peak": hbm, "unit": "GB/s", "frac": ach / hbm,
                         "traffic": None,
                         "algorithmic": "28 B per ray (direction in, result out); traversal reads BVH "
                                        "records from L2, so the kernel is latency/L2 bound, not HBM bound",
                         "kernel_ms": ms_per_step},
            "clocks": clocks.summary(), "gpu_launches": args.steps, "bvh_build_ms": build_ms,
            "hit_fraction": hit_frac}
    if not args.no_e2e:
        # the plugin call with host arrays: QueryForNLOS(numpy, numpy) -> numpy
        h_o = cams_np.reshape(-1)
        h_d = np.ascontiguousarray(dirs_np).reshape(-1)
        app.QueryForNLOS(h_o, h_d)
        barrier()
        t0 = time.perf_counter()
        e2e_steps = max(2, min(args.steps, 3))
        for _ in range(e2e_steps):
            res = app.QueryForNLOS(h_o, h_d)
        e2e_s = (time.perf_counter() - t0) / e2e_steps
        assert res.shape == (total_rays * 4,)
        line["e2e"] = {"value": world * total_rays / e2e_s, "unit": "rays/s",
                       "h2d_bytes_per_step": h_o.nbytes + h_d.nbytes, "d2h_bytes_per_step": total_rays * 16,
                       "ms_per_step": e2e_s * 1e3, "steps": e2e_steps,
                       "path": "ray_query.RayQueryApp.QueryForNLOS with numpy arrays in and out (C ABI "
                               "mb_ray_query_f32), host wall clock"}
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O

        threads = os.cpu_count() or 1
        os.environ.setdefault("OMP_NUM_THREADS", str(threads))
        t0 = time.perf_counter()
        O.ray_query(v_np, f_np, cams_np[:1], dirs_np[:1, :64])
        per_ray = (time.perf_counter() - t0) / 64
        n = int(max(64, min(n_rays, args.cpu_seconds / max(per_ray, 1e-9))))
        t0 = time.perf_counter()
        O.ray_query(v_np, f_np, cams_np[:1], dirs_np[:1, :n])
        line["cpu_baseline"] = {"value": n / (time.perf_counter() - t0), "unit": "rays/s", "cores": threads,
                                "kind": "port", "sample": f"{n} rays of camera 0, brute force over all "
                                f"{f_np.shape[0]} faces (double, no acceleration structure: the reference's "
                                "own query is a Vulkan pipeline)"}
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------------------
# Laplace single-layer collocation workload
# ---------------------------------------------------------------------------------------
def main_laplace(args, rank, world, local_rank):
    level, radius, dts = WORKLOADS[args.workload]
    nf = 20 * 4 ** level
    pairs = float(nf) ** 2
    config = {"workload": args.workload, "mesh": f"icosphere L{level}, radius {radius}", "n_faces": nf,
              "system": "P0 single-layer collocation at centroids, V sigma = 1 (exact sigma = 1/a)",
              "rule": "7-point rule per source face; faces sharing a vertex with the collocation face in "
                      "closed form (FP64)", "matrix": f"[F, F] {dts}",
              "l2": f"A ({pairs * (4 if dts == 'f32' else 8) / 1e9:.2f} GB) > L2, rewritten every step",
              "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference has no collocation system "
                              "(its Laplace path is the Galerkin one; new capability)"}), flush=True)
        return
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    R = pkg.roofline
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl")
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    dt = torch.float32 if dts == "f32" else torch.float64
    v_np, f_np = pkg.meshes.icosphere(level, radius)
    verts = torch.tensor(v_np, dtype=dt, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    A = torch.empty((nf, nf), dtype=dt, device=dev)
    stream = torch.cuda.current_stream(dev)
    L = pkg.layers
    near = L.laplace_near_pairs(faces)  # mesh topology, computed once like the edge numbering

    def assemble(v, f):
        L.laplace_colloc_sl(v, f, out=A, near=near, check_indices=False)

    def barrier():
        if world > 1:
            torch.distributed.barrier()
        torch.cuda.synchronize(dev)

    for _ in range(args.warmup):
        assemble(verts, faces)
    barrier()
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    barrier()
    for e0, e1 in ev:
        e0.record(stream)
        assemble(verts, faces)
        e1.record(stream)
    barrier()
    clocks.stop()
    ms = [a.elapsed_time(b) for a, b in ev]
    total_ms = sum(ms)
    if world > 1:
        t = torch.tensor([total_ms], device=dev)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        total_ms = float(t.item())
    ms_per_step = total_ms / args.steps
    value = world * pairs / (ms_per_step / 1e3)
    peaks = R.measured_peaks(REPO)
    sm_max = float(peaks.get("sm_max_mhz", 2070.0))
    evals = pairs * 7.0
    flop = evals * R.LAPLACE_SL_FLOP_PER_EVAL
    kern_s = statistics.mean(ms) / 1e3
    fp32_peak = R.fp32_peak_tflops(sm_max)
    hbm = float(peaks.get("hbm_gbs", 6800.0))
    out_bytes = pairs * (4 if dts == "f32" else 8)
    peak = fp32_peak if dts == "f32" else R.FP64_NOMINAL_TFLOPS
    line = {"metric": "collocation-matrix face pairs/s", "value": value, "unit": "pairs/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": dts, "data": "synthetic", "config": config,
            "roofline": {"bound": "fp32" if dts == "f32" else "fp64",
                         "achieved": flop / kern_s / 1e12, "peak": peak, "unit": "TFLOP/s",
                         "frac": flop / kern_s / 1e12 / peak,
                         "peak_source": "derived FP32 SIMT peak at the max SM clock" if dts == "f32" else
                                        "nominal GB300 FP64 (no measured FP64 figure)",
                         "hbm": {"achieved_gbs": out_bytes / kern_s / 1e9, "peak_gbs": hbm,
                                 "frac": out_bytes / kern_s / 1e9 / hbm},
                         "traffic": None,
                         "algorithmic": f"{R.LAPLACE_SL_FLOP_PER_EVAL} FLOP + {R.LAPLACE_MUFU_PER_EVAL} MUFU per "
                                        "evaluation x 7 evaluations per face pair x F^2; output "
                                        f"{4 if dts == 'f32' else 8} B per pair",
                         "kernel_ms": kern_s * 1e3},
            "clocks": clocks.summary(), "gpu_launches": args.steps}
    if not args.no_solve:
        ones = torch.ones(nf, dtype=torch.float64, device=dev)
        s0, s1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s0.record(stream)
        sigma, infos = pkg.mesh_MOM_3d.gmres_real(A, ones, restart=50, tol=1e-8, max_iters=1000)
        s1.record(stream)
        torch.cuda.synchronize(dev)
        err = float((sigma * radius - 1).abs().max())
        line["solve"] = {"what": "GMRES(50) to 1e-8 on V sigma = 1 (FP64 refinement residual)",
                         "gmres_ms": s0.elapsed_time(s1), "iterations": infos[0]["iterations"],
                         "rel_residual": infos[0]["rel_residual"], "converged": infos[0]["converged"],
                         "max_rel_err_sigma_vs_1_over_a": err,
                         "time_to_solution_ms": ms_per_step + s0.elapsed_time(s1)}
    if not args.no_e2e:
        h_v = torch.tensor(v_np, dtype=dt).pin_memory()
        h_f = torch.tensor(f_np, dtype=torch.int32).pin_memory()
        h_A = torch.empty((nf, nf), dtype=dt, pin_memory=True)
        d_v, d_f = torch.empty_like(verts), torch.empty_like(faces)

        def e2e_step():
            d_v.copy_(h_v, non_blocking=True)
            d_f.copy_(h_f, non_blocking=True)
            assemble(d_v, d_f)
            h_A.copy_(A, non_blocking=True)

        e2e_step()
        barrier()
        n_e2e = max(2, min(args.steps, 3))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(n_e2e):
            e2e_step()
        e1.record(stream)
        barrier()
        e2e_ms = e0.elapsed_time(e1) / n_e2e
        line["e2e"] = {"value": world * pairs / (e2e_ms / 1e3), "unit": "pairs/s",
                       "h2d_bytes_per_step": h_v.numel() * h_v.element_size() + h_f.numel() * 4,
                       "d2h_bytes_per_step": h_A.numel() * h_A.element_size(), "ms_per_step": e2e_ms,
                       "steps": n_e2e, "path": "layers.laplace_colloc_sl (C ABI mb_laplace_colloc_sl_*), pinned "
                                               "host mesh in, matrix back to pinned host memory"}
        del h_A
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O

        threads = os.cpu_count() or 1
        os.environ.setdefault("OMP_NUM_THREADS", str(threads))
        sub_level = max(1, level - 2)
        sv, sf = pkg.meshes.icosphere(sub_level, radius)
        t0 = time.perf_counter()
        O.laplace_colloc_sl(sv, sf)
        dt_cpu = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": float(sf.shape[0]) ** 2 / dt_cpu, "unit": "pairs/s", "cores": threads,
                                "kind": "port", "sample": f"the full collocation matrix of icosphere L{sub_level} "
                                f"({sf.shape[0]} faces) with the double C oracle (same rule); the reference has "
                                "no collocation path"}
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------------------
# many right-hand sides: tensor-core product + lockstep GMRES vs plain per-incidence GMRES
# ---------------------------------------------------------------------------------------
def main_radiate(args, rank, world, local_rank):
    """Scattered H on an observation grid from vertex currents (the post-processing step of the
    reference's MoM demo, demo_Helmholtz_MOM_3d.py:246-257)."""
    level, k, side = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    R = pkg.roofline
    config = {"workload": args.workload, "mesh": f"icosphere L{level}, radius 1", "ka": k,
              "field_points": f"{side} x {side} grid on the plane y = 0.05, x, z in [-3, 3]",
              "currents": "seeded complex vertex currents, vertex areas = sum of adjacent face areas / 3",
              "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference's radiation step is torch "
                              "tensor code inside its demo script; its algorithm is timed by cpu_baseline "
                              "(the C oracle)"}), flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    v_np, f_np = pkg.meshes.icosphere(level, 1.0)
    nv = v_np.shape[0]
    rng = np.random.default_rng(0)
    js_np = (rng.normal(size=(nv, 3)) + 1j * rng.normal(size=(nv, 3))).astype(np.complex64)
    tri = v_np[f_np]
    fa = 0.5 * np.linalg.norm(np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]), axis=1)
    va_np = np.zeros(nv)
    np.add.at(va_np, f_np.reshape(-1), np.repeat(fa / 3.0, 3))
    g1 = np.linspace(-3.0, 3.0, side)
    gx, gz = np.meshgrid(g1, g1, indexing="ij")
    pts_np = np.stack([gx.ravel(), 0.05 * np.ones(gx.size), gz.ravel()], -1).astype(np.float32)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    va = torch.tensor(va_np, dtype=torch.float32, device=dev)
    js = torch.tensor(js_np, device=dev)
    pts = torch.tensor(pts_np, device=dev)
    H = torch.empty((pts.shape[0], 3), dtype=torch.complex64, device=dev)
    M = pkg.mesh_MOM_3d
    pairs = float(pts.shape[0]) * nv
    stream = torch.cuda.current_stream(dev)
    for _ in range(args.warmup):
        M.radiate_H(pts, verts, va, js, k, out=H)
    torch.cuda.synchronize(dev)
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    torch.cuda.synchronize(dev)
    for e0, e1 in ev:
        e0.record(stream)
        M.radiate_H(pts, verts, va, js, k, out=H)
        e1.record(stream)
    torch.cuda.synchronize(dev)
    clocks.stop()
    ms = [a.elapsed_time(b) for a, b in ev]
    ms_per_step = sum(ms) / args.steps
    kern_s = statistics.mean(ms) / 1e3
    peaks = R.measured_peaks(REPO)
    sm_max = float(peaks.get("sm_max_mhz", 2070.0))
    fp32_peak, mufu_peak = R.fp32_peak_tflops(sm_max), R.mufu_peak_gops(sm_max)
    flop, mufu = pairs * R.RADIATE_FLOP_PER_PAIR, pairs * R.RADIATE_MUFU_PER_PAIR
    line = {"metric": "scattered-field (point, vertex) pairs/s", "value": world * pairs / (ms_per_step / 1e3),
            "unit": "pairs/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": ms_per_step, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic", "config": config,
            "roofline": {"bound": "fp32", "achieved": flop / kern_s / 1e12, "peak": fp32_peak, "unit": "TFLOP/s",
                         "frac": flop / kern_s / 1e12 / fp32_peak, "traffic": None,
                         "peak_source": "derived FP32 SIMT peak at the max SM clock",
                         "mufu": {"achieved_gops": mufu / kern_s / 1e9, "peak_gops": mufu_peak,
                                  "frac": mufu / kern_s / 1e9 / mufu_peak},
                         "algorithmic": f"{R.RADIATE_FLOP_PER_PAIR} FLOP + {R.RADIATE_MUFU_PER_PAIR} MUFU per "
                                        "(field point, vertex) pair",
                         "kernel": "radiate_h_kernel<float>", "kernel_ms": kern_s * 1e3},
            "clocks": clocks.summary(), "gpu_launches": args.steps}
    if not args.no_e2e:
        h_p = torch.tensor(pts_np).pin_memory()
        h_j = torch.tensor(js_np).pin_memory()
        h_H = torch.empty((pts.shape[0], 3), dtype=torch.complex64, pin_memory=True)
        d_p, d_j = torch.empty_like(pts), torch.empty_like(js)

        def e2e_step():
            d_p.copy_(h_p, non_blocking=True)
            d_j.copy_(h_j, non_blocking=True)
            M.radiate_H(d_p, verts, va, d_j, k, out=H)
            h_H.copy_(H, non_blocking=True)

        e2e_step()
        torch.cuda.synchronize(dev)
        n_e2e = max(2, min(args.steps, 3))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(n_e2e):
            e2e_step()
        e1.record(stream)
        torch.cuda.synchronize(dev)
        e2e_ms = e0.elapsed_time(e1) / n_e2e
        line["e2e"] = {"value": world * pairs / (e2e_ms / 1e3), "unit": "pairs/s",
                       "h2d_bytes_per_step": h_p.numel() * 4 + h_j.numel() * 8,
                       "d2h_bytes_per_step": h_H.numel() * 8, "ms_per_step": e2e_ms, "steps": n_e2e,
                       "path": "mesh_MOM_3d.radiate_H (C ABI mb_radiate_h_f32), pinned field points and "
                               "currents in, H back to pinned host memory"}
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O

        n_s = 4096
        threads = os.cpu_count() or 1
        os.environ.setdefault("OMP_NUM_THREADS", str(threads))
        sel = np.linspace(0, pts_np.shape[0] - 1, n_s).astype(np.int64)
        t0 = time.perf_counter()
        O.radiate_h(pts_np[sel].astype(np.float64), v_np, va_np, js_np.astype(np.complex128), k)
        dt_cpu = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": n_s * float(nv) / dt_cpu, "unit": "pairs/s", "cores": threads,
                                "kind": "port",
                                "sample": f"{n_s} of the {pts_np.shape[0]} field points against all {nv} vertices, "
                                          "double C oracle of the reference's formula (functions.py:844-868)"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def main_topology(args, rank, world, local_rank):
    """Mesh topology on the GPU: get_edge_unique (mesh_utils.py:921-977), the near-pair list
    (the nonzeros of compute_panel_relation, mesh_utils.py:700-725, built in O(F)) and the
    Z-row -> face-edge-row map of the edge-ordered assembly."""
    (level,) = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    U, M = pkg.utils, pkg.mesh_MOM_3d
    v_np, f_np = pkg.meshes.icosphere(level, 1.0)
    nf, nv = f_np.shape[0], v_np.shape[0]
    config = {"workload": args.workload, "mesh": f"icosphere L{level}", "n_faces": nf, "n_verts": nv,
              "outputs": "edges [E, 2], face-edge map [3F], edge faces [E, 2], near pairs [n, 2], Z-row map [2E + 1]",
              "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "topology is not the headline path; its CPU "
                              "run is the cpu_baseline of this workload"}), flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)

    def topo(v, f):
        edges, fei, adj = U.get_edge_unique(v, f)
        pairs = U.shared_vertex_pairs(f, v.shape[0])
        er = torch.empty(2 * edges.shape[0] + 1, dtype=torch.int32, device=f.device)
        pkg._lib.call("mb_mom_edge_rows", pkg._lib.ptr(fei), f.shape[0], edges.shape[0], pkg._lib.ptr(er),
                      pkg._lib.stream_of(f))
        return edges, fei, adj, pairs, er

    stream = torch.cuda.current_stream(dev)
    for _ in range(args.warmup):
        out = topo(verts, faces)
    torch.cuda.synchronize(dev)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    clocks = ClockSampler(dev.index)
    clocks.start()
    for e0, e1 in ev:
        e0.record(stream)
        out = topo(verts, faces)
        e1.record(stream)
    torch.cuda.synchronize(dev)
    clocks.stop()
    ms = [a.elapsed_time(b) for a, b in ev]
    ms_per_step = sum(ms) / args.steps
    edges, fei, adj, pairs, er = out
    ne, npairs = int(edges.shape[0]), int(pairs.shape[0])
    io_bytes = 12 * nf + 8 * ne + 12 * nf + 8 * ne + 8 * npairs + 4 * (2 * ne + 1)
    hbm = float(pkg.roofline.measured_peaks(REPO).get("hbm_gbs", 6800.0))
    line = {"metric": "mesh-topology faces/s", "value": world * nf / (ms_per_step / 1e3), "unit": "faces/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32 / int64",
            "data": "synthetic", "config": config, "n_edges": ne, "near_pairs": npairs,
            "roofline": {"bound": "hbm", "achieved": io_bytes / (ms_per_step / 1e3) / 1e9, "peak": hbm,
                         "unit": "GB/s", "frac": io_bytes / (ms_per_step / 1e3) / 1e9 / hbm, "traffic": None,
                         "algorithmic": "faces in + every output written once (sort passes not counted)",
                         "note": "sort / unique based (torch), latency-bound at this size"},
            "clocks": clocks.summary(), "gpu_launches": None}
    if not args.no_e2e:
        h_f = torch.tensor(f_np, dtype=torch.int32).pin_memory()
        d_f = torch.empty_like(faces)

        def e2e_step():
            d_f.copy_(h_f, non_blocking=True)
            res = topo(verts, d_f)
            return [t.to("cpu", non_blocking=True) for t in res]

        e2e_step()
        torch.cuda.synchronize(dev)
        n_e2e = max(2, min(args.steps, 3))
        t0 = time.perf_counter()
        for _ in range(n_e2e):
            outs = e2e_step()
        torch.cuda.synchronize(dev)
        e2e_s = (time.perf_counter() - t0) / n_e2e
        line["e2e"] = {"value": world * nf / e2e_s, "unit": "faces/s", "h2d_bytes_per_step": h_f.numel() * 4,
                       "d2h_bytes_per_step": sum(t.numel() * t.element_size() for t in outs),
                       "ms_per_step": e2e_s * 1e3, "steps": n_e2e,
                       "path": "utils.get_edge_unique + utils.shared_vertex_pairs + mb_mom_edge_rows, faces from "
                               "pinned host memory, every output back to the host"}
    if rank == 0 and not args.no_cpu_baseline:
        vc, fc = torch.tensor(v_np), torch.tensor(f_np, dtype=torch.int32)
        t0 = time.perf_counter()
        U.get_edge_unique(vc, fc)
        U.shared_vertex_pairs(fc)
        dt_cpu = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": nf / dt_cpu, "unit": "faces/s", "cores": torch.get_num_threads(),
                                "kind": "port", "sample": "the same unique-edge and near-pair construction with "
                                "torch on the host (the reference's get_edge_unique is this torch.unique; its "
                                "near pairs come from the dense O(F^2) relation, infeasible at this size)"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def main_lapref(args, rank, world, local_rank):
    """The reference's own Laplace path as demo_Laplace_3d.py drives it: MeshBEMSolver3d with
    the reference rule (double Duffy collapse, integrations_3d.py:252-452), P1, all-Dirichlet
    data, through solve (mesh_BEM_solver_3d.py:197-373): the shared-vertex relation, V and K
    panels, their packing, the right-hand side and the dense LU solve."""
    level, gq, radius = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    R, U = pkg.roofline, pkg.utils
    v_np, f_np = pkg.meshes.icosphere(level, radius)
    nf, nv = f_np.shape[0], v_np.shape[0]
    config = {"workload": args.workload, "mesh": f"icosphere L{level}, radius {radius}", "n_faces": nf,
              "n_verts": nv, "problem": "u = z on the whole surface (Dirichlet), unknown du/dn = z / a",
              "rule": f"the reference's (gaussQR = {gq}: collapsed Gauss rule per sub-domain), P1, float32",
              "solver": "dense LU (torch.linalg.solve), as the reference", "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference's Laplace path is torch code; its "
                              "algorithm is timed by cpu_baseline (the C oracle)"}), flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    z = verts[:, 2:3].clone()
    flags = torch.full((1, nv, 1), int(pkg.BoundaryType.DIRICHLET), dtype=torch.uint8, device=dev)
    g, h = z[None], torch.zeros_like(z)[None]
    solver = pkg.MeshBEMSolver3d(gaussQR=gq, order_type=1, BEM_type=int(pkg.BEMType.LAPLACE), wavenumber=1.0,
                                 logger=None, dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream(dev)
    for _ in range(args.warmup):
        out = solver.solve(verts, faces, g, h, flags)
    torch.cuda.synchronize(dev)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    calls0 = pkg._lib.call_count
    for e0, e1 in ev:
        e0.record(stream)
        out = solver.solve(verts, faces, g, h, flags)
        e1.record(stream)
    torch.cuda.synchronize(dev)
    clocks.stop()
    abi_calls = pkg._lib.call_count - calls0
    ms = [a.elapsed_time(b) for a, b in ev]
    ms_per_step = sum(ms) / args.steps
    neu = out[0][0]
    err = float(torch.linalg.norm(neu - z / radius) / torch.linalg.norm(z / radius))

    def timed(fn, reps=3):
        fn()
        torch.cuda.synchronize(dev)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(reps):
            r = fn()
        b.record(stream)
        torch.cuda.synchronize(dev)
        return a.elapsed_time(b) / reps, r

    areas = U.compute_face_areas(vertices=verts, faces=faces, keepdim=True).contiguous()
    normals = U.compute_face_normals(vertices=verts, faces=faces).contiguous()
    t_rel, rel = timed(lambda: U.compute_panel_relation(faces))
    rands = torch.cat((solver.single_layer.r1, solver.single_layer.r2), dim=-1)
    w = solver.single_layer.gauss_weights

    def panels(layer):
        return pkg.double_integration_on_panels_3d(int(pkg.BEMType.LAPLACE), 1, verts, faces, areas, normals, w, w,
                                                   rands, rands, rel, 1.0, layer)

    t_v, Vp = timed(lambda: panels(1))
    t_k, _ = timed(lambda: panels(2))
    t_pack, Vt = timed(lambda: U.pack_matrix_tight(1, Vp, verts, faces))
    rhs = torch.ones(nv, 1, device=dev)
    t_lu, _ = timed(lambda: torch.linalg.solve(Vt, rhs))
    del Vp
    # evaluations per face pair of the reference rule: separated pairs use the plain tensor
    # rule (n_w points on each face), the few pairs sharing a vertex their sub-domain tables
    n_w = int(w.numel())
    peaks = R.measured_peaks(REPO)
    fp32_peak = R.fp32_peak_tflops(float(peaks.get("sm_max_mhz", 2070.0)))
    hbm = float(peaks.get("hbm_gbs", 6800.0))
    flop = float(nf) ** 2 * n_w * n_w * (R.LAPLACE_SL_FLOP_PER_EVAL + 6)
    out_bytes = float(nf) ** 2 * 36
    line = {"metric": "Laplace Dirichlet solve time (reference rule)", "value": ms_per_step, "unit": "ms",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step,
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": config, "accuracy": {"dudn_rel_err": err,
                                           "note": "the reference rule's own discretisation error (double Duffy "
                                                   "collapse, no vertex alignment of the singular sub-domains)"},
            "breakdown_ms": {"panel_relation": t_rel, "V_panels": t_v, "K_panels": t_k, "pack_one_operator": t_pack,
                             "lu_solve_VxV": t_lu},
            "roofline": {"kernel": "laplace_panels_pair2_kernel<3, 1> + laplace_near_rows_kernel (V panels)", "bound": "fp32 / hbm",
                         "achieved": flop / (t_v / 1e3) / 1e12, "peak": fp32_peak, "unit": "TFLOP/s",
                         "frac": flop / (t_v / 1e3) / 1e12 / fp32_peak,
                         "peak_source": "derived FP32 SIMT peak at the max SM clock",
                         "hbm": {"achieved_gbs": out_bytes / (t_v / 1e3) / 1e9, "peak_gbs": hbm,
                                 "frac": out_bytes / (t_v / 1e3) / 1e9 / hbm},
                         "traffic": None,
                         "algorithmic": f"{n_w} x {n_w} evaluations per separated pair, "
                                        f"{R.LAPLACE_SL_FLOP_PER_EVAL} + 6 (P1 weights) FLOP and 1 rsqrt each; "
                                        "output 36 B per pair",
                         "kernel_ms": t_v},
            "clocks": clocks.summary(), "gpu_launches": abi_calls,
            "gpu_launches_note": "C-ABI calls in the timed region (each launches one or two of the library's "
                                 "kernels); torch's LU kernels not counted"}
    if not args.no_e2e:
        h_v = torch.tensor(v_np, dtype=torch.float32).pin_memory()
        h_f = torch.tensor(f_np, dtype=torch.int32).pin_memory()
        h_in = [t.cpu().pin_memory() for t in (g, h, flags)]
        h_out = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True) for t in out]
        d_v, d_f = torch.empty_like(verts), torch.empty_like(faces)
        d_in = [torch.empty_like(t) for t in (g, h, flags)]

        def e2e_step():
            d_v.copy_(h_v, non_blocking=True)
            d_f.copy_(h_f, non_blocking=True)
            for d, hh in zip(d_in, h_in):
                d.copy_(hh, non_blocking=True)
            res = solver.solve(d_v, d_f, *d_in)
            for hh, r in zip(h_out, res):
                hh.copy_(r, non_blocking=True)

        e2e_step()
        torch.cuda.synchronize(dev)
        n_e2e = max(2, min(args.steps, 3))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(n_e2e):
            e2e_step()
        e1.record(stream)
        torch.cuda.synchronize(dev)
        e2e_ms = e0.elapsed_time(e1) / n_e2e
        line["e2e"] = {"value": e2e_ms, "unit": "ms",
                       "h2d_bytes_per_step": h_v.numel() * 4 + h_f.numel() * 4 +
                                             sum(t.numel() * t.element_size() for t in h_in),
                       "d2h_bytes_per_step": sum(t.numel() * t.element_size() for t in h_out),
                       "ms_per_step": e2e_ms, "steps": n_e2e,
                       "path": "MeshBEMSolver3d.solve, reference rule (C ABI mb_panel_relation, "
                               "mb_laplace_panels_f32, mb_pack_tight_f32), pinned host mesh and data in, both traces "
                               "back"}
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O

        threads = os.cpu_count() or 1
        os.environ.setdefault("OMP_NUM_THREADS", str(threads))
        n_s = min(nf, 1024)
        a_np, n_np = areas.cpu().double().numpy(), normals.cpu().double().numpy()
        rel_np, r_np, w_np = rel.cpu().numpy(), rands.cpu().double().numpy(), w.cpu().double().numpy()
        t0 = time.perf_counter()
        O.laplace_panels(v_np, f_np, a_np, n_np, r_np, w_np, rel_np, 1, 1, rows=(0, n_s))
        O.laplace_panels(v_np, f_np, a_np, n_np, r_np, w_np, rel_np, 2, 1, rows=(0, n_s))
        t_ops = (time.perf_counter() - t0) * nf / n_s
        An = np.random.default_rng(0).normal(size=(nv, nv)) + nv * np.eye(nv)
        t0 = time.perf_counter()
        np.linalg.solve(An, np.ones(nv))
        t_solve = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": (t_ops + t_solve) * 1e3, "unit": "ms", "cores": threads, "kind": "port",
                                "sample": f"V and K panels of the first {n_s} of {nf} face rows with the double C "
                                          "restatement of the reference rule, scaled to all rows, plus a numpy LU "
                                          f"solve of size {nv}; packing not counted"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def main_lappanels(args, rank, world, local_rank):
    """The reference's Laplace operator assembly (double_integration_on_panels_3d,
    integrations_3d.py:252-452, as SingleLayer3d / DoubleLayer3d call it from
    mesh_BEM_solver_3d.py): V and K panels [F, F, 3, 3], P1, the reference rule, with the
    shared-vertex relation computed once per mesh like the solver does.  A step is both
    operators."""
    level, gq, radius = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    R, U = pkg.roofline, pkg.utils
    v_np, f_np = pkg.meshes.icosphere(level, radius)
    nf = f_np.shape[0]
    pairs = float(nf) ** 2
    config = {"workload": args.workload, "mesh": f"icosphere L{level}, radius {radius}", "n_faces": nf,
              "rule": f"the reference's (gaussQR = {gq}: collapsed Gauss rule per sub-domain), P1, float32",
              "output": "V and K panels [F, F, 3, 3] float32 (2 x 36 B per face pair)",
              "l2": f"outputs {2 * pairs * 36 / 1e9:.2f} GB per step > L2", "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference's Laplace path is torch code; its "
                              "algorithm is timed by cpu_baseline (the C oracle)"}), flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    areas = U.compute_face_areas(vertices=verts, faces=faces, keepdim=True).contiguous()
    normals = U.compute_face_normals(vertices=verts, faces=faces).contiguous()
    rel = U.compute_panel_relation(faces)
    p1, w1 = U.get_gaussion_integration_points_and_weights(gq, device=dev)
    rands, w = U.collapsed_rule_2d(p1, w1)
    stream = torch.cuda.current_stream(dev)

    def panels(layer, v=verts, f=faces, a=areas, n=normals, r=rel):
        return pkg.double_integration_on_panels_3d(int(pkg.BEMType.LAPLACE), 1, v, f, a, n, w, w, rands, rands, r,
                                                   1.0, layer)

    def step():
        return panels(1), panels(2)

    for _ in range(max(args.warmup, 3)):
        step()
    replica_barrier(world, dev)
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True),
           torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    calls0 = pkg._lib.call_count
    replica_barrier(world, dev)
    for e0, e1, e2 in ev:
        e0.record(stream)
        vp = panels(1)
        e1.record(stream)
        kp = panels(2)
        e2.record(stream)
        del vp, kp
    replica_barrier(world, dev)
    clocks.stop()
    abi_calls = pkg._lib.call_count - calls0
    step_ms = [a.elapsed_time(c) for a, _, c in ev]
    v_ms = statistics.mean(a.elapsed_time(b) for a, b, _ in ev)
    ms_per_step = replica_max(sum(step_ms), world, dev) / args.steps
    value = world * 2 * pairs / (ms_per_step / 1e3)
    # roofline: the V call (packed tiled kernel + near-pair kernel), separated pairs 16
    # evaluations of 15 + 6 FLOP and 1 rsqrt, 36 B written per pair
    n_w = int(w.numel())
    peaks = R.measured_peaks(REPO)
    fp32_peak = R.fp32_peak_tflops(float(peaks.get("sm_max_mhz", 2070.0)))
    hbm = float(peaks.get("hbm_gbs", 6800.0))
    flop = pairs * n_w * n_w * (R.LAPLACE_SL_FLOP_PER_EVAL + 6)
    out_bytes = pairs * 36
    traffic = None
    prof = os.path.join(REPO, "profiles", f"{args.workload}_traffic.json")
    if os.path.exists(prof):
        with open(prof) as fh:
            traffic = json.load(fh).get("dram_bytes_per_launch")
    line = {"metric": "Laplace panel pairs/s (V and K, reference rule)", "value": value, "unit": "pairs/s",
            "n_gpus": world, "steps": args.steps, "warmup": max(args.warmup, 3), "ms_per_step": ms_per_step,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": config,
            "roofline": {"kernel": "laplace_panels_pair2_kernel<3, 1> + laplace_near_rows_kernel (V panels)",
                         "bound": "hbm", "achieved": out_bytes / (v_ms / 1e3) / 1e9, "peak": hbm, "unit": "GB/s",
                         "frac": out_bytes / (v_ms / 1e3) / 1e9 / hbm, "traffic": traffic,
                         "algorithmic": "36 B written per face pair (nine float32 panel entries)",
                         "fp32": {"achieved_tflops": flop / (v_ms / 1e3) / 1e12, "peak_tflops": fp32_peak,
                                  "frac": flop / (v_ms / 1e3) / 1e12 / fp32_peak,
                                  "algorithmic": f"{n_w} x {n_w} evaluations per pair, "
                                                 f"{R.LAPLACE_SL_FLOP_PER_EVAL} + 6 (P1 weights) FLOP each"},
                         "kernel_ms": v_ms, "peak_source": "MEASURED_PEAKS.json hbm_gbs (burst copy)"},
            "clocks": clocks.summary(), "gpu_launches": 2 * abi_calls,
            "gpu_launches_note": "two kernels per C-ABI panel call (tiled + near pairs)"}
    if not args.no_e2e:
        h_v = torch.tensor(v_np, dtype=torch.float32).pin_memory()
        h_f = torch.tensor(f_np, dtype=torch.int32).pin_memory()
        h_out = [torch.empty((nf, nf, 3, 3), dtype=torch.float32, pin_memory=True) for _ in range(2)]
        d_v, d_f = torch.empty_like(verts), torch.empty_like(faces)

        def e2e_step():
            d_v.copy_(h_v, non_blocking=True)
            d_f.copy_(h_f, non_blocking=True)
            a = U.compute_face_areas(vertices=d_v, faces=d_f, keepdim=True).contiguous()
            n = U.compute_face_normals(vertices=d_v, faces=d_f).contiguous()
            r = U.compute_panel_relation(d_f)
            for hh, layer in zip(h_out, (1, 2)):
                hh.copy_(panels(layer, d_v, d_f, a, n, r), non_blocking=True)

        e2e_step()
        torch.cuda.synchronize(dev)
        n_e2e = max(2, min(args.steps, 3))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(n_e2e):
            e2e_step()
        e1.record(stream)
        torch.cuda.synchronize(dev)
        e2e_ms = e0.elapsed_time(e1) / n_e2e
        line["e2e"] = {"value": world * 2 * pairs / (e2e_ms / 1e3), "unit": "pairs/s",
                       "h2d_bytes_per_step": h_v.numel() * 4 + h_f.numel() * 4,
                       "d2h_bytes_per_step": sum(t.numel() * 4 for t in h_out), "ms_per_step": e2e_ms,
                       "steps": n_e2e,
                       "path": "double_integration_on_panels_3d (C ABI mb_panel_relation, mb_laplace_panels_f32) "
                               "from a pinned host mesh, both operators back to pinned host memory"}
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O

        threads = os.cpu_count() or 1
        n_s = min(nf, 512)
        a_np, n_np = areas.cpu().double().numpy(), normals.cpu().double().numpy()
        rel_np, r_np, w_np = rel.cpu().numpy(), rands.cpu().double().numpy(), w.cpu().double().numpy()
        t0 = time.perf_counter()
        O.laplace_panels(v_np, f_np, a_np, n_np, r_np, w_np, rel_np, 1, 1, rows=(0, n_s))
        O.laplace_panels(v_np, f_np, a_np, n_np, r_np, w_np, rel_np, 2, 1, rows=(0, n_s))
        t_cpu = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": 2 * n_s * nf / t_cpu, "unit": "pairs/s", "cores": threads, "kind": "port",
                                "sample": f"V and K panels of the first {n_s} of {nf} face rows with the double C "
                                          "restatement of the reference rule"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def main_pressure(args, rank, world, local_rank):
    """The ferrofluid pressure projection, MeshPressure.solve (src/mesh_ferrofluid/
    mesh_pressure.py:54-163): curvature, boundary data, the mixed Laplace solve and the
    velocity update, on a unit-sphere droplet resting on a solid (y <= 0: Neumann)."""
    (level,) = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    v_np, f_np = pkg.meshes.icosphere(level, 1.0)
    nf, nv = f_np.shape[0], v_np.shape[0]
    g, rho, dt = 9.8, 2.0, 0.01
    config = {"workload": args.workload, "mesh": f"icosphere L{level}, radius 1", "n_faces": nf, "n_verts": nv,
              "data": f"hydrostatic: vel = (0, g dt, 0), rho = {rho}, g = {g}, dt = {dt}, surface tension 0.07; "
                      "air (Dirichlet) for y > 0, solid (Neumann) below",
              "solver": "MeshPressure(rule dunavant7, solver schur), float32", "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference's pressure solve cannot run (its "
                              "hypersingular layer is None); the oracle's operators are timed by cpu_baseline"}),
                  flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    mp = pkg.MeshPressure(density_fluid=rho, gravity_strength=g, surface_tension=0.07, contact_angle=0.0,
                          gaussQR=3, order_type=1, logger=None, device=dev, dtype=torch.float32, solver="schur")
    flags = torch.where(verts[:, 1:2] > 0, int(pkg.BoundaryType.DIRICHLET), int(pkg.BoundaryType.NEUMANN))
    flags = flags.to(torch.uint8)[None]
    vel = torch.zeros((1, nv, 3), dtype=torch.float32, device=dev)
    vel[..., 1] = g * dt
    stream = torch.cuda.current_stream(dev)
    for _ in range(args.warmup):
        new = mp.solve(verts, faces, dt, vel, flags)
    torch.cuda.synchronize(dev)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    calls0 = pkg._lib.call_count
    for e0, e1 in ev:
        e0.record(stream)
        new = mp.solve(verts, faces, dt, vel, flags)
        e1.record(stream)
    torch.cuda.synchronize(dev)
    clocks.stop()
    abi_calls = pkg._lib.call_count - calls0
    ms_per_step = sum(a.elapsed_time(b) for a, b in ev) / args.steps
    n = pkg.utils.compute_vert_normals(verts, faces)
    solid = flags[0, :, 0] == int(pkg.BoundaryType.NEUMANN)
    vn = float((new[0] * n).sum(-1)[solid].abs().max()) / (g * dt)
    line = {"metric": "pressure projection step time", "value": ms_per_step, "unit": "ms", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic", "config": config,
            "accuracy": {"max_normal_velocity_on_solid_over_g_dt": vn},
            "roofline": {"kernel": "the mixed Laplace solve inside (laplace_mixed_* workloads)", "bound": None,
                         "achieved": None, "peak": None, "unit": None, "frac": None, "traffic": None},
            "clocks": clocks.summary(), "gpu_launches": abi_calls,
            "gpu_launches_note": "C-ABI calls in the timed region (each launches one or two of the library's "
                                 "kernels); torch's kernels not counted"}
    if not args.no_e2e:
        h_v = torch.tensor(v_np, dtype=torch.float32).pin_memory()
        h_f = torch.tensor(f_np, dtype=torch.int32).pin_memory()
        h_vel, h_flags = vel.cpu().pin_memory(), flags.cpu().pin_memory()
        h_new = torch.empty(new.shape, dtype=new.dtype, pin_memory=True)
        d_v, d_f, d_vel, d_flags = (torch.empty_like(t) for t in (verts, faces, vel, flags))

        def e2e_step():
            d_v.copy_(h_v, non_blocking=True)
            d_f.copy_(h_f, non_blocking=True)
            d_vel.copy_(h_vel, non_blocking=True)
            d_flags.copy_(h_flags, non_blocking=True)
            h_new.copy_(mp.solve(d_v, d_f, dt, d_vel, d_flags), non_blocking=True)

        e2e_step()
        torch.cuda.synchronize(dev)
        n_e2e = max(2, min(args.steps, 3))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(n_e2e):
            e2e_step()
        e1.record(stream)
        torch.cuda.synchronize(dev)
        e2e_ms = e0.elapsed_time(e1) / n_e2e
        line["e2e"] = {"value": e2e_ms, "unit": "ms",
                       "h2d_bytes_per_step": (h_v.numel() + h_f.numel() + h_vel.numel()) * 4 + h_flags.numel(),
                       "d2h_bytes_per_step": h_new.numel() * 4, "ms_per_step": e2e_ms, "steps": n_e2e,
                       "path": "MeshPressure.solve, pinned host mesh, velocities and flags in, new velocities back"}
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O

        threads = os.cpu_count() or 1
        os.environ.setdefault("OMP_NUM_THREADS", str(threads))
        n_s = min(nf, 1024)
        t0 = time.perf_counter()
        O.laplace_sym(v_np, f_np, 1, 1, rows=(0, n_s))
        O.laplace_sym(v_np, f_np, 2, 1, rows=(0, n_s))
        O.laplace_sym(v_np, f_np, 1, 0, rows=(0, n_s))
        t_ops = (time.perf_counter() - t0) * nf / n_s
        An = np.random.default_rng(0).normal(size=(nv, nv)) + nv * np.eye(nv)
        t0 = time.perf_counter()
        np.linalg.solve(An, np.ones(nv))
        t_solve = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": (t_ops + t_solve) * 1e3, "unit": "ms", "cores": threads, "kind": "port",
                                "sample": f"V, K and V0 panels of the first {n_s} of {nf} face rows with the double "
                                          f"C oracle, scaled to all rows, plus a numpy LU solve of size {nv} (the "
                                          "projection's curvature and gradients not counted)"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def main_lapmixed(args, rank, world, local_rank):
    """Mixed Dirichlet / Neumann Laplace solve through MeshBEMSolver3d.solve (the reference's
    facade, mesh_BEM_solver_3d.py:197-373): symmetric-rule V, K and hypersingular D,
    packed P1 matrices, the block system [[V, -K], [K', D]] and its dense solve."""
    level, dts = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    R, L, U = pkg.roofline, pkg.layers, pkg.utils
    v_np, f_np = pkg.meshes.icosphere(level, 1.0)
    nf, nv = f_np.shape[0], v_np.shape[0]
    config = {"workload": args.workload, "mesh": f"icosphere L{level}, radius 1", "n_faces": nf, "n_verts": nv,
              "problem": "u = z: Dirichlet data on z > 0, Neumann data du/dn = z on z <= 0",
              "rule": "dunavant7 (7 x 7 points, pairs sharing a vertex in closed form, FP64)",
              "operators": f"V, K, D packed [V, V] {dts} straight from the face pairs (no [F, F, 3, 3] panels)",
              "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference's Neumann / mixed branches never "
                              "run (its hypersingular layer is None); the oracle's operators are timed by "
                              "cpu_baseline"}), flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    dt = torch.float32 if dts == "f32" else torch.float64
    verts = torch.tensor(v_np, dtype=dt, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    z = verts[:, 2:3].clone()
    D_, N_ = int(pkg.BoundaryType.DIRICHLET), int(pkg.BoundaryType.NEUMANN)
    flags = torch.where(z > 0, D_, N_).to(torch.uint8)[None]
    g = torch.where(z > 0, z, 0.0)[None]
    h = torch.where(z > 0, 0.0, z)[None]
    solver = pkg.MeshBEMSolver3d(gaussQR=3, order_type=1, BEM_type=int(pkg.BEMType.LAPLACE), wavenumber=1.0,
                                 logger=None, dtype=dt, device=dev, rule="dunavant7", solver="schur")
    config["solver"] = ("schur: Cholesky factors of V on the Dirichlet vertices and of the Schur complement "
                        "D + K V^-1 K^T on the Neumann ones (cuSOLVER / cuBLAS through torch)")
    stream = torch.cuda.current_stream(dev)
    for _ in range(args.warmup):
        out = solver.solve(verts, faces, g, h, flags)
    torch.cuda.synchronize(dev)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    calls0 = pkg._lib.call_count
    for e0, e1 in ev:
        e0.record(stream)
        out = solver.solve(verts, faces, g, h, flags)
        e1.record(stream)
    torch.cuda.synchronize(dev)
    clocks.stop()
    abi_calls = pkg._lib.call_count - calls0
    ms = [a.elapsed_time(b) for a, b in ev]
    ms_per_step = sum(ms) / args.steps
    neu, dirv = out
    lower = (z <= 0).reshape(-1)
    far = (z > 0.3).reshape(-1)
    err_u = float(torch.linalg.norm(dirv[0][lower] - z[lower]) / torch.linalg.norm(z[lower]))
    err_t = float(torch.linalg.norm(neu[0][far] - z[far]) / torch.linalg.norm(z[far]))

    # per-stage times (the same calls solve() makes, timed one by one)
    def timed(fn, reps=3):
        fn()
        torch.cuda.synchronize(dev)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(reps):
            r = fn()
        b.record(stream)
        torch.cuda.synchronize(dev)
        return a.elapsed_time(b) / reps, r

    t_near, near = timed(lambda: U.shared_vertex_pairs(faces, nv))
    t_v, Vt = timed(lambda: L.laplace_sym_tight(verts, faces, 1, near))
    t_k, Kt = timed(lambda: L.laplace_sym_tight(verts, faces, 2, near))
    t_d, Dt = timed(lambda: L.laplace_sym_tight(verts, faces, 3, near))
    t_vp, Vp = timed(lambda: L.laplace_sym_panels(verts, faces, 1, 1, near))
    t_pack, _ = timed(lambda: U.pack_matrix_tight(1, Vp, verts, faces))
    del Vp
    is_d, is_n = (z > 0).reshape(-1), (z <= 0).reshape(-1)
    ks = Kt.transpose(0, 1)
    A = torch.cat((torch.cat((Vt[is_d][:, is_d], -ks[is_d][:, is_n]), 1),
                   torch.cat((ks.transpose(0, 1)[is_n][:, is_d], Dt[is_n][:, is_n]), 1)), 0)
    rhs = torch.ones(nv, 1, dtype=dt, device=dev)
    nd = int(is_d.sum())
    t_lu, _ = timed(lambda: torch.linalg.solve(A, rhs))
    SM = importlib.import_module("mesh-ferrofluid_gb300.mesh_BEM_solver_3d")
    t_schur, _ = timed(lambda: SM._schur_solve(Vt[is_d][:, is_d], ks[is_d][:, is_n], Dt[is_n][:, is_n],
                                               rhs[:nd, 0], rhs[nd:, 0]))
    peaks = R.measured_peaks(REPO)
    sm_max = float(peaks.get("sm_max_mhz", 2070.0))
    fp32_peak = R.fp32_peak_tflops(sm_max)
    flop_v = float(nf) ** 2 * 49 * R.LAPLACE_SYM_P1_FLOP_PER_EVAL
    ach = flop_v / (t_v / 1e3) / 1e12
    line = {"metric": "mixed Dirichlet/Neumann solve time", "value": ms_per_step, "unit": "ms",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step,
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": dts, "data": "synthetic",
            "config": config,
            "accuracy": {"u_rel_err_neumann_part": err_u, "dudn_rel_err_dirichlet_part_z_gt_0.3": err_t},
            "breakdown_ms": {"near_pairs": t_near, "V_packed": t_v, "K_packed": t_k, "D_packed": t_d,
                             "schur_solve_blocks": t_schur,
                             "not_on_the_path": {"V_panels": t_vp, "pack_V_panels": t_pack,
                                                 "lu_solve_block_system": t_lu}},
            "roofline": {"kernel": "lap_sym_pairs_kernel<1> + lap_sym_near_kernel (packed V)",
                         "bound": "fp32" if dts == "f32" else "fp64", "achieved": ach,
                         "peak": fp32_peak if dts == "f32" else R.FP64_NOMINAL_TFLOPS, "unit": "TFLOP/s",
                         "frac": ach / (fp32_peak if dts == "f32" else R.FP64_NOMINAL_TFLOPS),
                         "peak_source": "derived FP32 SIMT peak at the max SM clock",
                         "traffic": None,
                         "algorithmic": f"{R.LAPLACE_SYM_P1_FLOP_PER_EVAL} FLOP + 1 rsqrt per evaluation x 49 "
                                        "evaluations per face pair x F^2 (near pairs counted as separated); the "
                                        "packed path stores no panels (HBM traffic: mesh + 3 V reductions per row)",
                         "kernel_ms": t_v},
            "clocks": clocks.summary(), "gpu_launches": abi_calls,
            "gpu_launches_note": "C-ABI calls in the timed region (each launches one or two of the library's "
                                 "kernels); torch's sort / unique / LU kernels not counted"}
    if not args.no_e2e:
        h_v = torch.tensor(v_np, dtype=dt).pin_memory()
        h_f = torch.tensor(f_np, dtype=torch.int32).pin_memory()
        h_in = [t.cpu().pin_memory() for t in (g, h, flags)]
        h_out = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True) for t in out]
        d_v, d_f = torch.empty_like(verts), torch.empty_like(faces)
        d_in = [torch.empty_like(t) for t in (g, h, flags)]

        def e2e_step():
            d_v.copy_(h_v, non_blocking=True)
            d_f.copy_(h_f, non_blocking=True)
            for d, hh in zip(d_in, h_in):
                d.copy_(hh, non_blocking=True)
            res = solver.solve(d_v, d_f, *d_in)
            for hh, r in zip(h_out, res):
                hh.copy_(r, non_blocking=True)

        e2e_step()
        torch.cuda.synchronize(dev)
        n_e2e = max(2, min(args.steps, 3))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(n_e2e):
            e2e_step()
        e1.record(stream)
        torch.cuda.synchronize(dev)
        e2e_ms = e0.elapsed_time(e1) / n_e2e
        line["e2e"] = {"value": e2e_ms, "unit": "ms",
                       "h2d_bytes_per_step": h_v.numel() * h_v.element_size() + h_f.numel() * 4 +
                                             sum(t.numel() * t.element_size() for t in h_in),
                       "d2h_bytes_per_step": sum(t.numel() * t.element_size() for t in h_out),
                       "ms_per_step": e2e_ms, "steps": n_e2e,
                       "path": "MeshBEMSolver3d.solve (C ABI mb_laplace_sym_tight_*), pinned host mesh and boundary "
                               "data in, both traces back"}
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O

        threads = os.cpu_count() or 1
        os.environ.setdefault("OMP_NUM_THREADS", str(threads))
        n_s = min(nf, 1024)
        rows = (0, n_s)
        t0 = time.perf_counter()
        O.laplace_sym(v_np, f_np, 1, 1, rows=rows)
        O.laplace_sym(v_np, f_np, 2, 1, rows=rows)
        O.laplace_sym(v_np, f_np, 1, 0, rows=rows)
        t_ops = (time.perf_counter() - t0) * nf / n_s
        An = np.random.default_rng(0).normal(size=(nv, nv)) + nv * np.eye(nv)
        t0 = time.perf_counter()
        np.linalg.solve(An, np.ones(nv))
        t_solve = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": (t_ops + t_solve) * 1e3, "unit": "ms", "cores": threads, "kind": "port",
                                "sample": f"V, K and V0 panels of the first {n_s} of {nf} face rows with the double "
                                          f"C oracle (same rule), scaled to all rows, plus a numpy LU solve of "
                                          f"size {nv}; D from V0 and the packing not counted"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def main_mrhs(args, rank, world, local_rank):
    level, k, ndir = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    M = pkg.mesh_MOM_3d
    nrhs = 2 * ndir
    efie = args.workload.endswith("_efie")
    config = {"workload": args.workload, "mesh": f"ellipsoid 1.0/0.7/0.5 from icosphere L{level}, normal jitter "
              "N(0, 0.01 mean edge), seed 0", "ka": k, "rhs": f"{ndir} Fibonacci directions x 2 orthogonal "
              "polarisations",
              "formulation": ("EFIE, 7-point rule, closed-form singular pairs (FP64)" if efie else
                              "the reference's EFIE + MFIE operator and collapsed Gauss rule (gaussQR 4), its "
                              "excitation <f, E + n x H> for each plane wave"),
              "solve": "lockstep GMRES(50), every step one split-TF32x3 tcgen05 product with all right-hand sides",
              "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference solves one right-hand side per "
                              "dense LU and has no symmetric-rule EFIE; its own algorithm is timed by mom_ref_*"}),
                  flush=True)
        return
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl")
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    v_np, f_np = pkg.meshes.ellipsoid(level)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    edges, fei, _ = pkg.utils.get_edge_unique(verts, faces)
    ne = int(edges.shape[0])
    config["n_edges"] = ne
    dirs = pkg.meshes.fibonacci_lattice(ndir)
    ref_axis = np.where(np.abs(dirs[:, 2:3]) < 0.9, [[0.0, 0.0, 1.0]], [[1.0, 0.0, 0.0]])
    p1 = np.cross(dirs, ref_axis)
    p1 /= np.linalg.norm(p1, axis=1, keepdims=True)
    p2 = np.cross(dirs, p1)
    waves = M.plane_waves(k, np.concatenate([dirs, dirs]), np.concatenate([p1, p2]), device=dev)
    near = M.near_pairs(faces) if efie else None
    if not efie:
        areas = pkg.utils.compute_face_areas(verts, faces).contiguous()
        normals = pkg.utils.compute_face_normals(verts, faces).contiguous()
        px, wx = pkg.utils.get_gaussion_integration_points_and_weights(4, device=dev)
        py, wy = pkg.utils.get_gaussion_integration_points_and_weights(3, device=dev)
    stream = torch.cuda.current_stream(dev)
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731
    tol = 1e-5

    def solve_new():
        e = [ev() for _ in range(5)]
        e[0].record(stream)
        if efie:
            Z = M.assemble_Z_rwg_sym(verts, faces, fei, ne, k, pairs=near, check_indices=False)
            B = M.assemble_rhs_rwg_sym(verts, faces, fei, ne, waves)
        else:
            Z = M.assemble_Z_rwg(verts, faces, areas, normals, fei, ne, px, wx, py, wy, k, check_indices=False)
            B = M.assemble_rhs_rwg(verts, faces, areas, normals, fei, ne, px, wx, waves)
        e[1].record(stream)
        split = M.split_tf32(Z)
        e[2].record(stream)
        X, info = M.gmres_multi(split, B, restart=50, tol=tol, max_iters=3000)
        e[3].record(stream)
        torch.cuda.synchronize(dev)
        return Z, B, X, info, [e[0].elapsed_time(e[1]), e[1].elapsed_time(e[2]), e[2].elapsed_time(e[3])]

    for _ in range(max(1, min(args.warmup, 1))):
        Z, B, X, info, _ = solve_new()
    barrier = (lambda: (torch.distributed.barrier(), torch.cuda.synchronize(dev))) if world > 1 else \
        (lambda: torch.cuda.synchronize(dev))
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    runs = []
    for _ in range(args.steps):
        barrier()
        Z, B, X, info, parts = solve_new()
        runs.append(parts)
    clocks.stop()
    tot = [sum(p) for p in runs]
    ms = statistics.mean(tot)
    if world > 1:
        t = torch.tensor([ms], device=dev)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        ms = float(t.item())
    # accuracy against the FP64 dense solution (outside the timed region)
    Zd = Z.to(torch.complex128)
    Xref = torch.linalg.solve(Zd, B.to(torch.complex128))
    err_new = (torch.linalg.norm(X - Xref, dim=0) / torch.linalg.norm(Xref, dim=0)).cpu()
    # the plain path: one GMRES per incidence with HBM-bound FP32 matvecs, timed on a sample
    sample = list(range(0, nrhs, max(1, nrhs // 32)))
    e0, e1 = ev(), ev()
    e0.record(stream)
    errs_plain, iters_plain = [], []
    for c in sample:
        x1, inf1 = M.gmres(Z, B[:, c], restart=50, tol=tol, max_iters=3000)
        iters_plain.append(inf1[0]["iterations"])
        errs_plain.append((torch.linalg.norm(x1 - Xref[:, c]) / torch.linalg.norm(Xref[:, c])).item())
    e1.record(stream)
    torch.cuda.synchronize(dev)
    plain_ms_per_rhs = e0.elapsed_time(e1) / len(sample)
    asm_ms = statistics.mean(p[0] for p in runs)
    plain_total = asm_ms + plain_ms_per_rhs * nrhs
    # tensor-core product alone (the dominant kernel), for the roofline
    split = M.split_tf32(Z)
    X32 = X.to(torch.complex64)
    ws = torch.empty(M.cgemm_workspace_bytes(ne, nrhs), dtype=torch.uint8, device=dev)
    Y = torch.empty_like(X32)
    for _ in range(3):
        M.multi_rhs_matmul(split, X32, out=Y, workspace=ws)
    g0, g1 = ev(), ev()
    g0.record(stream)
    for _ in range(10):
        M.multi_rhs_matmul(split, X32, out=Y, workspace=ws)
    g1.record(stream)
    torch.cuda.synchronize(dev)
    gemm_ms = g0.elapsed_time(g1) / 10
    alg = 8.0 * ne * ne * nrhs
    peaks = pkg.roofline.measured_peaks(REPO)
    tf32_peak = float(peaks.get("bf16_tflops", 1900.0)) / 2.0
    line = {"metric": "incidences solved per second (assembly + solve to 1e-5 relative residual)",
            "value": world * nrhs / (ms / 1e3), "unit": "rhs/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32 (split-tf32x3 products, complex64 basis, FP64 Hessenberg and iterate)", "data": "synthetic",
            "config": config,
            "breakdown_ms": {"assembly_Z_and_B": asm_ms, "split": statistics.mean(p[1] for p in runs),
                             "gmres_multi": statistics.mean(p[2] for p in runs)},
            "solve": {"arnoldi_steps": info["iterations"], "restarts": info["restarts"],
                      "max_rel_residual": info["max_rel_residual"], "converged": info["converged"],
                      "max_rel_err_J_vs_fp64_lu": float(err_new.max()),
                      "median_rel_err_J_vs_fp64_lu": float(err_new.median())},
            "plain_path": {"what": "per-incidence GMRES(50), FP32 matvec, same tolerance, timed on "
                                   f"{len(sample)} of {nrhs} incidences and scaled",
                           "ms_per_rhs": plain_ms_per_rhs, "median_iterations": statistics.median(iters_plain),
                           "max_rel_err_J": max(errs_plain), "time_to_solution_ms": plain_total},
            "speedup_vs_plain": plain_total / ms,
            "roofline": {"bound": "tensor", "kernel": "tc_gemm_tf32x3_kernel (Z X, all right-hand sides)",
                         "achieved": 3 * alg / (gemm_ms / 1e3) / 1e12, "peak": tf32_peak, "unit": "TFLOP/s",
                         "frac": 3 * alg / (gemm_ms / 1e3) / 1e12 / tf32_peak, "traffic": None,
                         "algorithmic": f"8 E^2 m = {alg:.3e} FLOP per product; executed 3x (split TF32)",
                         "algorithmic_tflops": alg / (gemm_ms / 1e3) / 1e12, "kernel_ms": gemm_ms,
                         "peak_source": "TF32 dense = half the measured bf16 dense rate (MEASURED_PEAKS.json)"},
            "clocks": clocks.summary(), "gpu_launches": None}
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)


def main_cgemm(args, rank, world, local_rank):
    """Y = Z X on the tensor cores (split TF32 x 3) for E unknowns and m right-hand sides."""
    n, m, _ = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    M = pkg.mesh_MOM_3d
    config = {"workload": args.workload, "E": n, "m": m, "operands": "random complex64 Z [E, E], X [E, m]",
              "l2": "Z split (2 x 8 E^2 bytes) > L2", "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference has no multi-right-hand-side "
                              "product (one dense LU per right-hand side)"}), flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    g = torch.Generator(device=dev).manual_seed(0)
    Z = torch.complex(torch.randn(n, n, device=dev, generator=g), torch.randn(n, n, device=dev, generator=g))
    X = torch.complex(torch.randn(n, m, device=dev, generator=g), torch.randn(n, m, device=dev, generator=g))
    split = M.split_tf32(Z)
    del Z
    ws = torch.empty(M.cgemm_workspace_bytes(n, m), dtype=torch.uint8, device=dev)
    Y = torch.empty(n, m, dtype=torch.complex64, device=dev)
    M.multi_rhs_matmul(split, X, out=Y, workspace=ws, check=True)
    for _ in range(args.warmup):
        M.multi_rhs_matmul(split, X, out=Y, workspace=ws)
    torch.cuda.synchronize(dev)
    stream = torch.cuda.current_stream(dev)
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        M.multi_rhs_matmul(split, X, out=Y, workspace=ws)
    e1.record(stream)
    torch.cuda.synchronize(dev)
    clocks.stop()
    ms = e0.elapsed_time(e1) / args.steps
    alg = 8.0 * n * n * m
    peaks = pkg.roofline.measured_peaks(REPO)
    tf32_peak = float(peaks.get("bf16_tflops", 1900.0)) / 2.0
    line = {"metric": "complex multi-RHS product, algorithmic TFLOP/s (8 E^2 m per product)",
            "value": alg / (ms / 1e3) / 1e12, "unit": "TFLOP/s", "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32 (split-tf32x3, FP32 accumulation)", "data": "synthetic",
            "config": config,
            "roofline": {"bound": "tensor", "achieved": 3 * alg / (ms / 1e3) / 1e12, "peak": tf32_peak,
                         "unit": "TFLOP/s", "frac": 3 * alg / (ms / 1e3) / 1e12 / tf32_peak, "traffic": None,
                         "algorithmic": "3 x 8 E^2 m executed TF32 FLOP per product",
                         "peak_source": "TF32 dense = half the measured bf16 dense rate (MEASURED_PEAKS.json)"},
            "clocks": clocks.summary(), "gpu_launches": 2 * args.steps}
    if rank == 0:
        print(json.dumps(line), flush=True)


def batch_meshes(n_mesh, seed):
    """Star-shaped closed surfaces from icosphere levels 2-4, ka ~ U(1, 8), seeded."""
    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    rng = np.random.default_rng(seed)
    levels = rng.integers(2, 5, n_mesh)
    kas = rng.uniform(1.0, 8.0, n_mesh)
    meshes = [pkg.meshes.star_shape(int(levels[i]), seed=seed * 1000 + i) for i in range(n_mesh)]
    return meshes, [float(k) for k in kas], [int(l) for l in levels]


def main_batch(args, rank, world, local_rank):
    """Config 4: time to a TTS_TARGET relative error in J (every column) for all meshes and
    incidences of the batch, plain per-mesh path against the batched preconditioned path."""
    n_mesh, nc, seed = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    MM = pkg.mesh_MOM_3d
    meshes, ks, levels = batch_meshes(n_mesh, seed)
    efie = args.workload.endswith("_efie")
    formulation = "efie_sym" if efie else "cfie_ref"
    config = {"workload": args.workload, "meshes": f"{n_mesh} star-shaped surfaces r = 1 + sum of 6 real SH "
              "(l <= 4, amplitudes U(0, 0.15)) on icosphere levels 2-4", "ka": "U(1, 8)",
              "incidences_per_mesh": nc,
              "formulation": ("EFIE, 7-point rule, closed-form singular pairs (FP64)" if efie else
                              "the reference's EFIE + MFIE operator and collapsed Gauss rule (gaussQR 4)"),
              "levels": {str(l): levels.count(l) for l in (2, 3, 4)}, "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference handles one mesh per solver call "
                              "and has no symmetric-rule EFIE; its own algorithm is timed by mom_ref_*"}), flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    rng = np.random.default_rng(seed + 1)
    waves = []
    for i in range(n_mesh):
        d = rng.normal(size=(nc, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        p = np.cross(d, rng.normal(size=(nc, 3)))
        p /= np.linalg.norm(p, axis=1, keepdims=True)
        waves.append(MM.plane_waves(ks[i], d, p))
    waves = torch.stack(waves).to(dev)
    # the plain path is config 2's GMRES(50); the batched path restarts every 150 steps (near
    # interior resonances of the EFIE a few eigenvalues of the preconditioned operator sit near
    # zero and a 50-step cycle cannot capture them)
    restart, restart_b, cap = 50, 150, 20000
    bt = pkg.batch.MeshBatch(meshes, ks, device=dev, formulation=formulation)
    if not efie:
        px, wx = pkg.utils.get_gaussion_integration_points_and_weights(4, device=dev)
        py, wy = pkg.utils.get_gaussion_integration_points_and_weights(3, device=dev)
    config["unknowns"] = {"total": int(sum(bt.n_edges)), "min": int(min(bt.n_edges)), "max": int(max(bt.n_edges))}
    stream = torch.cuda.current_stream(dev)
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731
    z_flat = torch.zeros(bt.z_size, dtype=torch.complex64, device=dev)
    B = bt.excitation(waves)
    asm_cfg = bt.autotune_assembly(z_flat)  # assembly tile and block schedule, timed per candidate
    bt.assemble(out=z_flat)
    rows = bt.autotune(z_flat)
    P = bt.spai(z_flat)

    # FP64 reference J of every column (untimed)
    t0 = time.perf_counter()
    if efie:
        z64 = torch.zeros(bt.z_size, dtype=torch.complex128, device=dev)
        vd = bt.verts.double().contiguous()
        pkg._lib.call("mb_mom_sym_zmat_batched_c128", pkg._lib.ptr(vd), pkg._lib.ptr(bt.faces),
                      pkg._lib.ptr(bt.fei), pkg._lib.ptr(bt.desc), pkg._lib.ptr(bt.ks), bt.n_mesh, bt.total_blocks,
                      pkg._lib.ptr(bt.near), bt.near.shape[0], pkg._lib.ptr(z64), pkg._lib.stream_of(z64))
        b64 = torch.zeros((bt.n_rows, n_mesh * nc), dtype=torch.complex128, device=dev)
        wv = waves.to(torch.float64).contiguous()
        pkg._lib.call("mb_mom_sym_rhs_batched_c128", pkg._lib.ptr(vd), pkg._lib.ptr(bt.faces),
                      pkg._lib.ptr(bt.fei), pkg._lib.ptr(bt.desc), bt.n_mesh, bt.total_faces, pkg._lib.ptr(wv), nc,
                      n_mesh * nc, pkg._lib.ptr(b64), pkg._lib.stream_of(b64))
        ref_what = ("FP64 batched assembly (complex128 Z_i, FP64 quadrature and singular integrals), per-mesh FP64 "
                    "preconditioned GMRES (FP64 products) to a 1e-10 relative residual")
    else:
        ref_what = ("the FP32-assembled complex64 Z_i solved to a 1e-10 relative residual (compensated "
                    "refinement residual); an FP64 assembly of the reference rule is too slow at GB300's FP64 rate")
    # restart 100: near an interior resonance restarted GMRES(50) stagnates above 1e-10 even
    # in FP64 (one 64-mesh case stopped at the iteration cap with a 8.5e-4 error in J); every
    # reference column must report convergence
    refs = {}
    ref_worst_res = 0.0
    for i in range(n_mesh):
        e = bt.n_edges[i]
        o = int(bt.edge_offsets[i])
        Pi = MM.SpaiPreconditioner(P.cols[o:o + e], P.vals[o:o + e], 0)
        if efie:
            zi = bt.z_block(z64, i).contiguous()
            bi = b64[:e, nc * i:nc * (i + 1)]
        else:
            zi = bt.z_block(z_flat, i).contiguous()
            bi = B[:e, nc * i:nc * (i + 1)].to(torch.complex128)
        refs[i], rinfo = MM.pgmres(zi, bi, M=Pi, restart=100, tol=1e-10, max_iters=40000)
        if not all(q["converged"] for q in rinfo):
            raise RuntimeError(f"FP64 reference of mesh {i} did not converge: {rinfo}")
        ref_worst_res = max(ref_worst_res, max(q["rel_residual"] for q in rinfo))
    if efie:
        del z64, b64
    torch.cuda.synchronize(dev)
    ref_s = time.perf_counter() - t0

    def col_errs(X):  # relative error of J per column of mesh i, all meshes -> max
        worst = 0.0
        for i in range(n_mesh):
            e = bt.n_edges[i]
            d = torch.linalg.norm(X[:e, nc * i:nc * (i + 1)] - refs[i], dim=0) / torch.linalg.norm(refs[i], dim=0)
            worst = max(worst, float(d.max()))
        return worst

    # batched preconditioned path: calibrate the tolerance, then time it end to end
    def run_batched(tol, precond=True):
        e = [ev() for _ in range(4)]
        torch.cuda.synchronize(dev)
        e[0].record(stream)
        bt.assemble(out=z_flat)
        Bb = bt.excitation(waves)
        e[1].record(stream)
        Pb = bt.spai(z_flat) if precond else None
        e[2].record(stream)
        X, info = bt.solve(z_flat, Bb, restart=restart_b, tol=tol, max_iters=cap, use_graph=True, M=Pb)
        e[3].record(stream)
        torch.cuda.synchronize(dev)
        return X, info, e[0].elapsed_time(e[1]), e[1].elapsed_time(e[2]), e[2].elapsed_time(e[3])

    # per preconditioner choice (with / without the near-field SAI; the EFIE always takes it)
    # the loosest ladder tolerance that reaches the target, then the faster of the two (one
    # untimed run each).  Without the SAI the lockstep cycles restart from an FP32 residual,
    # which stalls near 1e-6: tighter tolerances are not tried.
    cands = {}
    for precond in ((True,) if efie else (True, False)):
        for tol in (TTS_LADDER if precond else [t for t in TTS_LADDER if t >= 1e-6]):
            X, info, *_ = run_batched(tol, precond)
            if col_errs(X) <= TTS_TARGET:
                r_ = run_batched(tol, precond)
                cands[precond] = (tol, r_[2] + r_[3] + r_[4])
                break
    if cands:
        use_pc = min(cands, key=lambda q: cands[q][1])
        chosen = cands[use_pc][0]
    else:
        use_pc, chosen = True, None
    for _ in range(max(1, min(args.warmup, 1))):
        run_batched(chosen or TTS_LADDER[-1], use_pc)
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    runs = [run_batched(chosen or TTS_LADDER[-1], use_pc) for _ in range(args.steps)]
    clocks.stop()
    X, info = runs[-1][0], runs[-1][1]
    asm_ms = statistics.mean(r[2] for r in runs)
    pc_ms = statistics.mean(r[3] for r in runs)
    solve_ms = statistics.mean(r[4] for r in runs)
    total_ms = asm_ms + pc_ms + solve_ms
    batched_err = col_errs(X)

    # plain path: each mesh assembled on its own, each incidence solved by GMRES(50) from zero
    # with FP32 products and no preconditioner; each column stops at the loosest tolerance of
    # the ladder that reaches the target (found beforehand, untimed)
    def mesh_system(i):
        v, f = meshes[i]
        vt = torch.tensor(np.asarray(v), dtype=torch.float32, device=dev)
        ft = torch.tensor(np.asarray(f), dtype=torch.int32, device=dev)
        edges, fei, _ = pkg.utils.get_edge_unique(vt, ft)
        ne = int(edges.shape[0])
        if efie:
            Z = MM.assemble_Z_rwg_sym(vt, ft, fei, ne, ks[i])
            Bi = MM.assemble_rhs_rwg_sym(vt, ft, fei, ne, waves[i])
        else:
            a = pkg.utils.compute_face_areas(vt, ft).contiguous()
            nn = pkg.utils.compute_face_normals(vt, ft).contiguous()
            Z = MM.assemble_Z_rwg(vt, ft, a, nn, fei, ne, px, wx, py, wy, ks[i])
            Bi = MM.assemble_rhs_rwg(vt, ft, a, nn, fei, ne, px, wx, waves[i])
        return Z, Bi

    plain_tol = {}
    plain_reached = True
    for i in range(n_mesh):
        Z, Bi = mesh_system(i)
        for r in range(nc):
            ref = refs[i][:, r]
            for tol in TTS_LADDER:
                x1, inf1 = MM.gmres(Z, Bi[:, r], restart=restart, tol=tol, max_iters=cap)
                if float((x1 - ref).norm() / ref.norm()) <= TTS_TARGET:
                    plain_tol[(i, r)] = tol
                    break
                if inf1[0]["iterations"] >= cap:  # tighter tolerances cannot do better within the cap
                    plain_tol[(i, r)] = tol
                    plain_reached = False
                    break
            else:
                plain_tol[(i, r)] = TTS_LADDER[-1]
                plain_reached = False
        del Z, Bi
    e0, e1 = ev(), ev()
    torch.cuda.synchronize(dev)
    e0.record(stream)
    plain_iters, plain_err = [], 0.0
    plain_X = {}
    for i in range(n_mesh):
        Z, Bi = mesh_system(i)
        xs = []
        for r in range(nc):
            x1, inf1 = MM.gmres(Z, Bi[:, r], restart=restart, tol=plain_tol[(i, r)], max_iters=cap)
            plain_iters.append(inf1[0]["iterations"])
            xs.append(x1)
        plain_X[i] = torch.stack(xs, 1)
        del Z, Bi
    e1.record(stream)
    torch.cuda.synchronize(dev)
    plain_ms = e0.elapsed_time(e1)
    for i in range(n_mesh):
        d = torch.linalg.norm(plain_X[i] - refs[i], dim=0) / torch.linalg.norm(refs[i], dim=0)
        plain_err = max(plain_err, float(d.max()))
    line = {"metric": "batch time to a 1e-4 relative error in J (every mesh and incidence), plain FP32 path vs "
                      "batched preconditioned path",
            "value": total_ms, "unit": "ms", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": total_ms, "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32 (FP64 near pairs, complex64 basis, FP64 Hessenberg and iterate)", "data": "synthetic",
            "config": config, "target_rel_err_J": TTS_TARGET, "reference_J": ref_what, "reference_J_seconds": ref_s,
            "reference_J_max_rel_residual": ref_worst_res,
            "batched": {"what": "1 assembly + 1 excitation launch for all meshes, the near-field SAI of every mesh "
                                "in one launch (when faster), lockstep (right-preconditioned) GMRES(150) on all "
                                "columns with the block-diagonal product (one CUDA graph per restart cycle)",
                        "preconditioned": use_pc,
                        "calibration_ms": {("sai" if q else "none"): v[1] for q, v in cands.items()},
                        "tol": chosen, "reached": chosen is not None and batched_err <= TTS_TARGET,
                        "assembly_and_excitation_ms": asm_ms, "precond_ms": pc_ms, "solve_ms": solve_ms,
                        "arnoldi_steps": info["iterations"], "restarts": info["restarts"],
                        "max_rel_residual": info["max_rel_residual"], "max_rel_err_J": batched_err,
                        "matvec_rows_per_warp": rows, "assembly_tile_schedule": asm_cfg,
                        "assembly_candidates_ms": {str(k): v for k, v in bt.asm_times.items()},
                        "precond_status": P.status if use_pc else None},
            "plain_path": {"what": "per mesh: FP32 assembly + excitation, then one GMRES(50) per incidence from zero "
                                   "(FP32 products, no preconditioner, mb_gmres_c64), each column at the loosest "
                                   "ladder tolerance that reaches the target (a column that hits the cap of "
                                   f"{cap} steps stops there: its time is a lower bound)",
                           "time_to_solution_ms": plain_ms, "reached": plain_reached,
                           "median_iterations": statistics.median(plain_iters), "max_iterations": max(plain_iters),
                           "max_rel_err_J": plain_err},
            "speedup_vs_plain": plain_ms / total_ms,
            "speedup_note": None if plain_reached else "the plain path did not reach the target on every column "
                            "within the cap; its time and this ratio are lower bounds",
            "clocks": clocks.summary(), "gpu_launches": None}
    if rank == 0:
        print(json.dumps(line), flush=True)


def _incidences(rng, n, nc, ks, MM):
    waves, dirs = [], []
    for i in range(n):
        d = rng.normal(size=(nc, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        p = np.cross(d, rng.normal(size=(nc, 3)))
        p /= np.linalg.norm(p, axis=1, keepdims=True)
        waves.append(MM.plane_waves(ks[i], d, p))
        dirs.append((d, p))
    return waves, dirs


def main_learned(args, rank, world, local_rank):
    """Generate solves, train the edge-graph network on them, and measure what its initial
    guess saves on held-out meshes (levels 2-3 of the batched-mesh distribution)."""
    n_train, n_test, nc = WORKLOADS[args.workload]
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    MM, L = pkg.mesh_MOM_3d, pkg.learned
    config = {"workload": args.workload, "train": f"{n_train} star-shaped meshes (levels 2-3) x {nc} incidences = "
              f"{n_train * nc} solves, ka ~ U(1, 8)", "test": f"{n_test} held-out meshes x {nc} incidences",
              "formulation": "the reference's EFIE + MFIE operator and rule", "network": f"{L.LAYERS} message-passing "
              f"layers, hidden {L.HIDDEN}, BF16 weights / activations, FP32 accumulation", "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference has no learned component"}),
                  flush=True)
        return
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)

    def mesh_set(n, seed):
        rng = np.random.default_rng(seed)
        levels = rng.integers(2, 4, n)
        ks = rng.uniform(1.0, 8.0, n)
        meshes = [pkg.meshes.star_shape(int(levels[i]), seed=seed * 100000 + i) for i in range(n)]
        waves, dirs = _incidences(rng, n, nc, ks, MM)
        return meshes, [float(k) for k in ks], waves, dirs

    def solve_chunks(meshes, ks, waves, tol, chunk=64, x0_fn=None, use_graph=True, aug_fn=None):
        """Per chunk: batch, assemble, excite, (initial guess or deflation subspace), solve.
        Yields per-chunk results."""
        for c0 in range(0, len(meshes), chunk):
            c1 = min(c0 + chunk, len(meshes))
            bt = pkg.batch.MeshBatch(meshes[c0:c1], ks[c0:c1], device=dev, formulation="cfie_ref")
            Z = bt.assemble()
            B = bt.excitation(torch.stack(waves[c0:c1]).to(dev))
            bt.rows_per_warp = 2
            X0 = x0_fn(bt, Z, B, c0) if x0_fn else None
            aug = aug_fn(bt, Z, B, c0) if aug_fn else None
            X, info = bt.solve(Z, B, restart=50, tol=tol, max_iters=2000, use_graph=use_graph, X0=X0, aug=aug)
            yield bt, Z, B, X, info, c0

    # 1. training data: solves by the batched solver
    t0 = time.perf_counter()
    meshes, ks, waves, dirs = mesh_set(n_train, 1)
    items = []
    graphs = {}
    for bt, Z, B, X, info, c0 in solve_chunks(meshes, ks, waves, 1e-6):
        for i in range(bt.n_mesh):
            mi = c0 + i
            v, f = meshes[mi]
            g = L.edge_graph(torch.tensor(v, dtype=torch.float32, device=dev),
                             torch.tensor(f, dtype=torch.int32, device=dev))
            for r in range(nc):
                b_e, j = bt.column(B, i, r), bt.column(X, i, r)
                x0 = L.node_features(g, ks[mi], dirs[mi][0][r], dirs[mi][1][r], b_e)
                items.append((g, x0, j))
    samples = L.build_samples(items)
    del items
    torch.cuda.synchronize(dev)
    gen_s = time.perf_counter() - t0
    # 2. training on the GPU kernels
    t0 = time.perf_counter()
    net = L.EdgeGNN(dev, seed=0)
    losses = L.train(net, samples, epochs=8, batch=32, lr=1e-3)
    torch.cuda.synchronize(dev)
    train_s = time.perf_counter() - t0
    del samples
    # 3. held-out meshes: GMRES from zero vs from the network's guess, tolerance 1e-4
    tmeshes, tks, twaves, tdirs = mesh_set(n_test, 2)

    tgraphs = {}

    def learned_x0(bt, Z, B, c0):
        """All columns of the chunk: batched features, one forward pass, then per column the
        residual-minimising combination over its mesh's predictions (a 2 nc-vector subspace)."""
        c1 = c0 + bt.n_mesh
        if c0 not in tgraphs:
            gs = [L.edge_graph(torch.tensor(tmeshes[mi][0], dtype=torch.float32, device=dev),
                               torch.tensor(tmeshes[mi][1], dtype=torch.int32, device=dev)) for mi in range(c0, c1)]
            tgraphs[c0] = L.batch_graph(gs)
        khat = np.stack([np.asarray(tdirs[mi][0], np.float32) for mi in range(c0, c1)])
        pol = np.stack([np.asarray(tdirs[mi][1], np.float32) for mi in range(c0, c1)])
        x0, nbr, flat = L.batch_node_features(tgraphs[c0], tks[c0:c1], khat, pol, B, nc)
        pred = net.predict(x0, nbr)
        return L.subspace_guess(bt, Z, B, pred, flat, nc)

    def learned_aug(bt, Z, B, c0):
        """Deflation subspace of every mesh, K = 16: the real and imaginary parts of the
        network's predicted currents for the mesh's nc incidences and for the same incidences
        with the orthogonal polarisation (k x p); the solver starts every cycle from their
        residual-minimising combination and runs its Arnoldi steps in the complement."""
        c1 = c0 + bt.n_mesh
        if c0 not in tgraphs:
            gs = [L.edge_graph(torch.tensor(tmeshes[mi][0], dtype=torch.float32, device=dev),
                               torch.tensor(tmeshes[mi][1], dtype=torch.int32, device=dev)) for mi in range(c0, c1)]
            tgraphs[c0] = L.batch_graph(gs)
        khat = np.stack([np.asarray(tdirs[mi][0], np.float32) for mi in range(c0, c1)])
        pol = np.stack([np.asarray(tdirs[mi][1], np.float32) for mi in range(c0, c1)])
        pol2 = np.cross(khat, pol)
        w2 = torch.stack([MM.plane_waves(tks[mi], khat[mi - c0].astype(np.float64), pol2[mi - c0].astype(np.float64))
                          for mi in range(c0, c1)]).to(dev)
        B2 = bt.excitation(w2)  # same nc: the batch's column layout is unchanged
        cols = []
        for p_, b_ in ((pol, B), (pol2, B2)):
            x0, nbr, flat = L.batch_node_features(tgraphs[c0], tks[c0:c1], khat, p_, b_, nc)
            P = torch.zeros(B.shape, dtype=torch.complex64, device=dev)
            P.view(-1)[flat] = net.predict(x0, nbr).to(torch.complex64)
            P3 = P.view(bt.n_rows, bt.n_mesh, nc)
            cols += [P3.real, P3.imag]
        U = torch.cat(cols, 2).to(torch.complex64)
        return bt.augmentation(Z, U)

    res = {}
    for name, fn, afn in (("zero_start", None, None), ("learned_start", learned_x0, None),
                          ("learned_deflation16", None, learned_aug)):
        for _ in range(2):  # second pass timed (first warms the caches and builds the graphs)
            steps, cols = [], []
            for bt, Z, B, X, info, c0 in solve_chunks(tmeshes, tks, twaves, 1e-4, x0_fn=fn, use_graph=False,
                                                      aug_fn=afn):
                steps.append(info["iterations"])
                cols.append(info["column_iterations"].cpu())
        # time of the whole held-out set (assembly + guess + solve)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for bt, Z, B, X, info, c0 in solve_chunks(tmeshes, tks, twaves, 1e-4, x0_fn=fn, use_graph=False, aug_fn=afn):
            pass
        e1.record()
        torch.cuda.synchronize(dev)
        colsteps = torch.cat(cols).double()
        res[name] = {"arnoldi_steps_per_chunk": steps, "total_steps": int(sum(steps)), "ms": e0.elapsed_time(e1),
                     "column_steps_mean": float(colsteps.mean()), "column_steps_median": float(colsteps.median()),
                     "column_steps_p90": float(torch.quantile(colsteps, 0.9))}
    # accuracy of the guess on the held-out set (relative error vs the 1e-6 solution)
    errs = []
    for bt, Z, B, X, info, c0 in solve_chunks(tmeshes[:64], tks[:64], twaves[:64], 1e-6):
        X0 = learned_x0(bt, Z, B, c0)
        num = torch.linalg.norm(X0.to(torch.complex128) - X, dim=0)
        errs.extend((num / torch.linalg.norm(X, dim=0)).cpu().tolist())
    line = {"metric": "held-out time to 1e-4 relative residual with the learned initial guess", "value":
            res["learned_start"]["ms"], "unit": "ms", "n_gpus": 1, "steps": 1, "warmup": 1,
            "ms_per_step": res["learned_start"]["ms"], "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "bf16 network, f32 solver", "data": "synthetic", "config": config,
            "generation_s": gen_s, "training_s": train_s, "epoch_losses": losses,
            "guess_rel_err_median": float(np.median(errs)), "guess_rel_err_p90": float(np.quantile(errs, 0.9)),
            "zero_start": res["zero_start"], "learned_start": res["learned_start"],
            "learned_deflation16": res["learned_deflation16"],
            "deflation_time_ratio": res["zero_start"]["ms"] / res["learned_deflation16"]["ms"],
            "deflation": "16 vectors per mesh (real and imaginary parts of the predicted currents for the mesh's "
                         "incidences and for their orthogonal polarisations), GCRO-style augmented lockstep GMRES "
                         "(mb_gmres_blockdiag_aug_c64)",
            "step_ratio": res["zero_start"]["total_steps"] / max(1, res["learned_start"]["total_steps"]),
            "column_step_ratio": res["zero_start"]["column_steps_mean"] / max(1e-9, res["learned_start"][
                "column_steps_mean"]),
            "guess": "least-squares combination of the real and imaginary parts of the network's predictions for "
                     "the mesh's incidences (2 nc vectors per mesh), per column",
            "time_ratio": res["zero_start"]["ms"] / res["learned_start"]["ms"], "gpu_launches": None}
    if rank == 0:
        print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------------------
# GPU arm
# ---------------------------------------------------------------------------------------
# ---------------------------------------------------------------------------------------
# time to a 1e-4 relative error in J: plain FP32 path against the mixed-precision path
# ---------------------------------------------------------------------------------------
TTS_TARGET = 1e-4
TTS_LADDER = (1e-3, 3e-4, 1e-4, 3e-5, 1e-5, 3e-6, 1e-6, 3e-7, 1e-7, 3e-8, 1e-8, 3e-9, 1e-9, 3e-10, 1e-10)


def time_to_solution(pkg, dev, level, k, sym, gq=4, Z=None, repeats=2):
    """Time to a TTS_TARGET relative error in J (the RWG edge coefficients, x-polarised plane
    wave along +z) against an FP64 reference J, for complete GPU paths, each run from the mesh
    on the device to the solution inside the timed region (CUDA events):

    * plain: the FP32 assembly + excitation, then GMRES(50) from zero with FP32 products and
      no preconditioner (mb_gmres_c64: host-driven Arnoldi, FP64 refinement residual);
    * plain_device: the same assembly, then the device-resident GMRES of the mixed path
      without its preconditioner (mb_pgmres_c64 with no M);
    * mixed_fp32 / mixed: the same FP32 assembly + excitation, the near-field sparse approximate
      inverse (mb_spai_build_c64), then right-preconditioned GMRES(50) with the restart cycle
      on the device as a CUDA graph (mb_pgmres_c64: complex64 basis, FP64 Hessenberg and iterate,
      compensated refinement residual); mixed reads a half-precision copy of Z in the Arnoldi
      products.

    Each path's stopping tolerance is the loosest of TTS_LADDER whose solution reaches the
    target (found by untimed solves on the same matrix); the timed runs' errors are reported.
    """
    import torch

    M = pkg.mesh_MOM_3d
    U = pkg.utils
    v_np, f_np = pkg.meshes.icosphere(level)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    edges, fei, _ = U.get_edge_unique(verts, faces)
    E = int(edges.shape[0])
    areas = U.compute_face_areas(verts, faces).contiguous()
    normals = U.compute_face_normals(verts, faces).contiguous()
    near = M.near_pairs(faces)
    pw = M.plane_waves(k, [[0.0, 0.0, 1.0]], [[1.0, 0.0, 0.0]], device=dev)
    if Z is None or tuple(Z.shape) != (E, E):
        Z = torch.empty((E, E), dtype=torch.complex64, device=dev)
    if not sym:
        px, wx = U.get_gaussion_integration_points_and_weights(gq, device=dev)
        py, wy = U.get_gaussion_integration_points_and_weights(gq - 1, device=dev)
        er = M.edge_rows(fei, faces.shape[0], E)

    def assemble():
        Z.zero_()
        if sym:
            M.assemble_Z_rwg_sym(verts, faces, fei, E, k, out=Z, pairs=near, check_indices=False)
            rhs = M.assemble_rhs_rwg_sym(verts, faces, fei, E, pw)
        else:
            M.assemble_Z_rwg(verts, faces, areas, normals, fei, E, px, wx, py, wy, k, out=Z, check_indices=False,
                             order="edges", edge_rows_map=er)
            rhs = M.assemble_rhs_rwg(verts, faces, areas, normals, fei, E, px, wx, pw)
        return rhs[:, 0].to(torch.complex128)

    def precond(half=False):
        P = M.spai_preconditioner(Z, verts, faces, fei, E, pairs=near)
        return (P, M.half_copy(Z)) if half else (P, None)

    def solve(path, b, tol, PH=(None, None)):
        if path == "plain":
            return M.gmres(Z, b, restart=50, tol=tol, max_iters=20000)
        if path == "plain_device":
            return M.pgmres(Z, b, M=None, restart=50, tol=tol, max_iters=20000, use_graph=True)
        return M.pgmres(Z, b, M=PH[0], restart=50, tol=tol, max_iters=20000, use_graph=True, Z_half=PH[1],
                        inner_rtol=3e-3)

    # FP64 reference J (untimed)
    t0 = time.perf_counter()
    b = assemble()
    P, Zh = precond(half=True)
    if sym:
        Z64 = M.assemble_Z_rwg_sym(verts.double(), faces, fei, E, k, pairs=near, check_indices=False)
        b64 = M.assemble_rhs_rwg_sym(verts.double(), faces, fei, E, pw)[:, 0]
        j_ref, rinfo = M.pgmres(Z64, b64, M=P, restart=50, tol=1e-12, max_iters=20000)
        del Z64, b64
        ref_what = ("FP64 assembly (complex128 Z: FP64 quadrature and closed-form singular integrals), FP64 "
                    "GMRES (FP64 products) to a 1e-12 relative residual")
    else:
        j_ref, rinfo = M.pgmres(Z, b, M=P, restart=50, tol=1e-12, max_iters=20000)
        ref_what = ("the FP32-assembled complex64 Z solved to a 1e-12 relative residual (an FP64 assembly of the "
                    "reference rule takes about a minute at GB300's FP64 rate at this size; the FP32 assembly's "
                    "own error is checked against the float64 oracle by the parity tests)")
    torch.cuda.synchronize(dev)
    ref_s = time.perf_counter() - t0
    if not rinfo[0]["converged"]:
        raise RuntimeError(f"FP64 reference J did not converge: {rinfo}")
    jn = float(j_ref.norm())

    def err(x):
        return float((x - j_ref).norm()) / jn

    out = {"target_rel_err_J": TTS_TARGET, "reference_J": ref_what,
           "reference_J_info": {"iterations": rinfo[0]["iterations"], "rel_residual": rinfo[0]["rel_residual"],
                                "seconds": ref_s},
           "mesh": f"icosphere L{level} ({faces.shape[0]} faces, {E} RWG unknowns)", "ka": k,
           "formulation": ("EFIE, 7-point rule on both triangles, closed-form FP64 near pairs" if sym else
                           f"reference CFIE (EFIE+MFIE), collapsed Gauss-Legendre gaussQR={gq}"),
           "excitation": "x-polarised unit plane wave along +z"}
    for path in ("plain", "plain_device", "mixed_fp32", "mixed"):
        chosen = None
        for tol in TTS_LADDER:
            x, inf = solve(path, b, tol, (P, Zh if path == "mixed" else None))
            e = err(x)
            if e <= TTS_TARGET:
                chosen = (tol, e, inf[0])
                break
        if chosen is None:
            out[path] = {"reached": False, "last_tol": TTS_LADDER[-1], "last_err": e, "last_info": inf[0]}
            continue
        tol = chosen[0]
        runs = []
        for _ in range(repeats):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
            torch.cuda.synchronize(dev)
            ev[0].record()
            bb = assemble()
            ev[1].record()
            PH = precond(half=path == "mixed") if path.startswith("mixed") else (None, None)
            ev[2].record()
            x, inf = solve(path, bb, tol, PH)
            ev[3].record()
            torch.cuda.synchronize(dev)
            runs.append({"total_ms": ev[0].elapsed_time(ev[3]), "assembly_ms": ev[0].elapsed_time(ev[1]),
                         "precond_ms": ev[1].elapsed_time(ev[2]), "solve_ms": ev[2].elapsed_time(ev[3]),
                         "iterations": inf[0]["iterations"], "restarts": inf[0]["restarts"],
                         "rel_residual": inf[0]["rel_residual"], "rel_err_J": err(x)})
        out[path] = {"reached": all(r["rel_err_J"] <= TTS_TARGET for r in runs), "tol": tol,
                     "ms": statistics.mean(r["total_ms"] for r in runs), "runs": runs}
    out["plain"]["what"] = ("FP32 assembly + excitation, GMRES(50) from zero with FP32 products and no "
                            "preconditioner, host-driven Arnoldi, FP64 refinement residual (mb_gmres_c64)")
    out["plain_device"]["what"] = ("FP32 assembly + excitation, the mixed path's device-resident GMRES(50) from "
                                   "zero without the preconditioner (mb_pgmres_c64, no M)")
    out["mixed_fp32"]["what"] = ("FP32 assembly + excitation, near-field SAI preconditioner (mb_spai_build_c64), "
                                 "right-preconditioned GMRES(50) with the restart cycle on the device as a CUDA "
                                 "graph, complex64 basis, compensated-FP32 refinement residual (mb_pgmres_c64)")
    out["mixed"]["what"] = ("as mixed_fp32, with the Arnoldi products on a half-precision copy of Z "
                            "(mb_half_copy_c64, made inside the timed region) and each inner cycle ended at a 3e-3 "
                            "reduction, refined against the complex64 residual")
    if out["mixed"].get("reached"):
        for p in ("plain", "plain_device", "mixed_fp32"):
            if out[p].get("reached"):
                out[f"ratio_{p}_over_mixed"] = out[p]["ms"] / out["mixed"]["ms"]
    del P, Zh, b, j_ref
    return out


def main_efie_solve(args, rank, world, local_rank):
    """The mixed-precision EFIE path of the time-to-solution comparison as its own workload:
    each step assembles Z (7-point rule, complex64, FP64 near pairs), builds the near-field SAI
    and the half-precision copy, and solves by right-preconditioned GMRES(50) to a 3e-5
    relative residual; the error in J against an FP64 solution is checked after the timing."""
    level, k = WORKLOADS[args.workload]
    config = {"workload": args.workload, "mesh": f"icosphere L{level}", "ka": k, "formulation": "EFIE, 7-point rule",
              "excitation": "x-polarised unit plane wave along +z", "parallelism": "replicas"}
    if args.impl == "reference":
        if rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "the reference has no symmetric-rule EFIE and "
                              "solves by dense LU; its own algorithm is timed by mom_ref_*"}), flush=True)
        return
    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    M = pkg.mesh_MOM_3d
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)
    v_np, f_np = pkg.meshes.icosphere(level)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    edges, fei, _ = pkg.utils.get_edge_unique(verts, faces)
    E = int(edges.shape[0])
    near = M.near_pairs(faces)
    pw = M.plane_waves(k, [[0.0, 0.0, 1.0]], [[1.0, 0.0, 0.0]], device=dev)
    Z = torch.empty((E, E), dtype=torch.complex64, device=dev)

    def step():
        Z.zero_()
        M.assemble_Z_rwg_sym(verts, faces, fei, E, k, out=Z, pairs=near, check_indices=False)
        b = M.assemble_rhs_rwg_sym(verts, faces, fei, E, pw)[:, 0].to(torch.complex128)
        P = M.spai_preconditioner(Z, verts, faces, fei, E, pairs=near)
        x, info = M.pgmres(Z, b, M=P, restart=50, tol=3e-5, max_iters=5000, Z_half=M.half_copy(Z),
                           inner_rtol=3e-3)
        return x, info

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize(dev)
    stream = torch.cuda.current_stream(dev)
    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        x, info = step()
    e1.record(stream)
    torch.cuda.synchronize(dev)
    clocks.stop()
    ms = e0.elapsed_time(e1) / args.steps
    err = None
    if not args.no_solve:  # the FP64 check (skipped when profiling the timed path alone)
        Z64 = M.assemble_Z_rwg_sym(verts.double(), faces, fei, E, k, pairs=near, check_indices=False)
        b64 = M.assemble_rhs_rwg_sym(verts.double(), faces, fei, E, pw)[:, 0]
        P = M.spai_preconditioner(Z, verts, faces, fei, E, pairs=near)
        j_ref, _ = M.pgmres(Z64, b64, M=P, restart=50, tol=1e-12, max_iters=20000)
        err = float((x - j_ref).norm() / j_ref.norm())
    line = {"metric": "time to a <1e-4 relative error in J, mixed-precision EFIE path", "value": ms, "unit": "ms",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32 assembly (FP64 near pairs), binary16 Arnoldi products, FP64 Hessenberg and iterate",
            "data": "synthetic", "config": config, "iterations": info[0]["iterations"],
            "restarts": info[0]["restarts"], "rel_residual": info[0]["rel_residual"], "rel_err_J_vs_fp64": err,
            "clocks": clocks.summary()}
    if rank == 0:
        print(json.dumps(line), flush=True)


def main():
    args = _args()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.workload.startswith("efie_solve_"):
        return main_efie_solve(args, rank, world, local_rank)
    if args.workload.startswith("ray_"):
        return main_rays(args, rank, world, local_rank)
    if args.workload.startswith("pressure_"):
        return main_pressure(args, rank, world, local_rank)
    if args.workload.startswith("laplace_mixed"):
        return main_lapmixed(args, rank, world, local_rank)
    if args.workload.startswith("laplace_panels"):
        return main_lappanels(args, rank, world, local_rank)
    if args.workload.startswith("laplace_ref"):
        return main_lapref(args, rank, world, local_rank)
    if args.workload.startswith("laplace_"):
        return main_laplace(args, rank, world, local_rank)
    if args.workload.startswith("mrhs_"):
        return main_mrhs(args, rank, world, local_rank)
    if args.workload.startswith("cgemm_"):
        return main_cgemm(args, rank, world, local_rank)
    if args.workload.startswith("batch_"):
        return main_batch(args, rank, world, local_rank)
    if args.workload.startswith("learned_"):
        return main_learned(args, rank, world, local_rank)
    if args.workload.startswith("radiate_"):
        return main_radiate(args, rank, world, local_rank)
    if args.workload.startswith("topology_"):
        return main_topology(args, rank, world, local_rank)
    level, k, gq = WORKLOADS[args.workload]
    n_faces = 20 * 4 ** level
    n_edges = 30 * 4 ** level
    pairs = float(n_faces) ** 2
    sym = gq == 0
    config = {"workload": args.workload, "mesh": f"icosphere L{level}", "n_faces": n_faces,
              "n_edges": n_edges, "ka": k,
              "rule": ("7-point degree-5 rule on both triangles; pairs sharing a vertex in FP64 with "
                       "closed-form 1/R integrals" if sym else
                       f"reference collapsed Gauss-Legendre gaussQR={gq} ({gq * gq} test x "
                       f"{(gq - 1) ** 2} source points, rotated per local edge)"),
              "formulation": "EFIE" if sym else "EFIE+MFIE (reference CFIE)",
              "output": "RWG Z [E,E] complex64",
              "l2": "Z (7.55 GB at L5) > L2, rewritten every step", "parallelism": "replicas"}

    if args.impl == "reference":
        if rank != 0:
            return
        if sym:
            print(json.dumps({"impl": "reference", "unavailable": "the reference has no symmetric-rule "
                              "EFIE with singularity extraction (new capability); its own algorithm is "
                              "timed by the mom_ref_* workloads"}), flush=True)
            return
        vals, info = cpu_sample_run(args.workload, args.cpu_seconds, steps=args.steps,
                                    warmup=min(args.warmup, 1))
        v = statistics.mean(vals)
        # a step of this arm is the bounded sample it times (the metric is a rate): ms_per_step
        # is that sample's wall time; the whole matrix at this rate is reported beside it
        line = {"metric": "Z-assembly triangle pairs/s", "value": v, "unit": "pairs/s",
                "impl": "reference", "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
                "ms_per_step": info["sample_ms_per_step"], "full_matrix_ms_at_this_rate": pairs / v * 1e3,
                "higher_is_better": True, "scaling": "weak",
                "vs_baseline": None, "dtype": "f32", "data": "synthetic", "config": config,
                "cpu_baseline": {"value": v, "unit": "pairs/s", **info},
                "e2e": {"value": v, "unit": "pairs/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line), flush=True)
        return

    import torch

    pkg = importlib.import_module("mesh-ferrofluid_gb300")
    R = pkg.roofline
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl")
    dev = torch.device("cuda", local_rank if world > 1 else 0)
    torch.cuda.set_device(dev)

    v_np, f_np = pkg.meshes.icosphere(level)
    verts = torch.tensor(v_np, dtype=torch.float32, device=dev)
    faces = torch.tensor(f_np, dtype=torch.int32, device=dev)
    edges, fei, _ = pkg.utils.get_edge_unique(verts, faces)
    areas = pkg.utils.compute_face_areas(verts, faces).contiguous()
    normals = pkg.utils.compute_face_normals(verts, faces).contiguous()
    if not sym:
        px, wx = pkg.utils.get_gaussion_integration_points_and_weights(gq, device=dev)
        py, wy = pkg.utils.get_gaussion_integration_points_and_weights(gq - 1, device=dev)
    Z = torch.zeros((n_edges, n_edges), dtype=torch.complex64, device=dev)
    stream = torch.cuda.current_stream(dev)
    M = pkg.mesh_MOM_3d
    near = M.near_pairs(faces) if sym else None
    n_near = int(near.shape[0]) if sym else 0
    er_map = None if sym else M.edge_rows(fei, faces.shape[0], n_edges)  # mesh preprocessing, like fei

    def assemble(out):
        if sym:
            M.assemble_Z_rwg_sym(verts, faces, fei, n_edges, k, out=out, pairs=near, check_indices=False)
        else:
            M.assemble_Z_rwg(verts, faces, areas, normals, fei, n_edges, px, wx, py, wy, k, out=out,
                             check_indices=False, order="edges", edge_rows_map=er_map)

    def step():
        Z.zero_()
        assemble(Z)

    def barrier():
        replica_barrier(world, dev)

    for _ in range(args.warmup):
        step()
    barrier()

    clocks = ClockSampler(dev.index)
    clocks.start()
    time.sleep(0.3)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True),
           torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    barrier()
    for e0, e1, e2 in ev:
        e0.record(stream)
        Z.zero_()
        e1.record(stream)
        assemble(Z)
        e2.record(stream)
    barrier()
    clocks.stop()
    step_ms = [a.elapsed_time(c) for a, _, c in ev]
    kern_ms = [b.elapsed_time(c) for _, b, c in ev]
    total_ms = replica_max(sum(step_ms), world, dev)  # the slowest replica
    ms_per_step = total_ms / args.steps
    value = world * pairs / (ms_per_step / 1e3)
    kern_avg_s = statistics.mean(kern_ms) / 1e3

    # roofline of the dominant kernel (assembly), per launch
    if sym:
        evals = (pairs - n_near) / 2 * 49.0  # each separated pair once for both orders (near pairs: FP64)
        flop = evals * R.EFIE_FLOP_PER_EVAL
        mufu = evals * R.EFIE_MUFU_PER_EVAL
        per_eval = f"{R.EFIE_FLOP_PER_EVAL} FLOP + {R.EFIE_MUFU_PER_EVAL} MUFU per evaluation x 49 " \
                   f"evaluations per unordered separated pair x (F^2 - {n_near} near pairs) / 2; kernel time = all kernels"
    else:
        evals = pairs * R.ref_rule_evals_per_pair(gq)
        flop = evals * R.CFIE_FLOP_PER_EVAL
        mufu = evals * R.CFIE_MUFU_PER_EVAL
        per_eval = f"{R.CFIE_FLOP_PER_EVAL} FLOP + {R.CFIE_MUFU_PER_EVAL} MUFU per evaluation x " \
                   f"{R.ref_rule_evals_per_pair(gq)} evaluations per pair x F^2 pairs"
    peaks = R.measured_peaks(REPO)
    sm_max = float(peaks.get("sm_max_mhz", 2070.0))
    fp32_peak = R.fp32_peak_tflops(sm_max)
    mufu_peak = R.mufu_peak_gops(sm_max)
    achieved = flop / kern_avg_s / 1e12
    traffic = None
    prof = os.path.join(REPO, "profiles", f"{args.workload}_traffic.json")
    if os.path.exists(prof):
        with open(prof) as fh:
            traffic = json.load(fh).get("dram_bytes_per_launch")
    roof = {"bound": "fp32", "achieved": achieved, "peak": fp32_peak, "unit": "TFLOP/s",
            "frac": achieved / fp32_peak, "traffic": traffic,
            "peak_source": f"152 SMs x 256 FP32 FLOP/clk x {sm_max:.0f} MHz (max SM clock of "
                           "MEASURED_PEAKS.json; the file has no FP32-SIMT figure)",
            "mufu": {"achieved_gops": mufu / kern_avg_s / 1e9, "peak_gops": mufu_peak,
                     "frac": mufu / kern_avg_s / 1e9 / mufu_peak},
            "algorithmic": per_eval,
            "kernel": ("sym_pairs_kernel + mom_sym_regular_rows_kernel + mom_sym_near_kernel" if sym else
                       f"mom_ref_zmat_edge_kernel<{gq},{gq - 1}> (Z row by Z row)"),
            "kernel_ms": kern_avg_s * 1e3}

    line = {"metric": "Z-assembly triangle pairs/s", "value": value, "unit": "pairs/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_per_step,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": config, "roofline": roof, "clocks": clocks.summary(),
            "gpu_launches": args.steps * (5 if sym else 1)}

    # time to a 1e-4 error in J, plain FP32 path vs the mixed-precision path (reported beside the
    # headline; both formulations on the same 30 720-unknown sphere for the default workload)
    if not args.no_solve:
        tts = {}
        if sym:
            tts["efie_7pt"] = time_to_solution(pkg, dev, level, k, True, Z=Z)
        else:
            tts["cfie_ref_rule"] = time_to_solution(pkg, dev, level, k, False, gq=gq, Z=Z)
            if level == 5:
                tts["efie_7pt"] = time_to_solution(pkg, dev, level, k, True, Z=Z)
        line["time_to_solution"] = tts

    # end to end through the public operator: host (pinned) inputs in, Z back to host memory
    if not args.no_e2e:
        h_verts = torch.tensor(v_np, dtype=torch.float32).pin_memory()
        h_faces = torch.tensor(f_np, dtype=torch.int32).pin_memory()
        h_fei = fei.cpu().pin_memory()
        h_rules = [] if sym else [t.cpu().pin_memory() for t in (px, wx, py, wy)]
        h_Z = torch.empty((n_edges, n_edges), dtype=torch.complex64, pin_memory=True)
        d_verts = torch.empty_like(verts)
        d_faces = torch.empty_like(faces)
        d_fei = torch.empty_like(fei)
        d_rules = [torch.empty_like(t, device=dev) for t in h_rules]

        def e2e_step():
            d_verts.copy_(h_verts, non_blocking=True)
            d_faces.copy_(h_faces, non_blocking=True)
            d_fei.copy_(h_fei, non_blocking=True)
            for d, h in zip(d_rules, h_rules):
                d.copy_(h, non_blocking=True)
            a = pkg.utils.compute_face_areas(d_verts, d_faces).contiguous()
            nn = pkg.utils.compute_face_normals(d_verts, d_faces).contiguous()
            if sym:
                # test faces in 16 ranges; finished Z rows drained to host while the next range runs
                M.assemble_Z_rwg_sym(d_verts, d_faces, d_fei, n_edges, k, out=Z, pairs=near,
                                     check_indices=False, out_host=h_Z, chunks=16)
            else:
                # Z rows assembled in 16 ranges, each range's copy to host overlapping the next
                M.assemble_Z_rwg(d_verts, d_faces, a, nn, d_fei, n_edges, *d_rules, k, out=Z,
                                 check_indices=False, out_host=h_Z, chunks=16)

        e2e_step()
        barrier()
        e2e_steps = max(2, min(args.steps, 3))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        barrier()
        e0.record(stream)
        for _ in range(e2e_steps):
            e2e_step()
        e1.record(stream)
        barrier()
        e2e_ms = e0.elapsed_time(e1) / e2e_steps
        h2d = (h_verts.numel() * 4 + h_faces.numel() * 4 + h_fei.numel() * 4
               + sum(t.numel() * 4 for t in h_rules))
        line["e2e"] = {"value": world * pairs / (e2e_ms / 1e3), "unit": "pairs/s",
                       "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": h_Z.numel() * 8,
                       "ms_per_step": e2e_ms, "steps": e2e_steps,
                       "path": ("mesh_MOM_3d.assemble_Z_rwg_sym(out_host=...) (C ABI "
                                "mb_mom_sym_zmat_rwg_to_host_c64: test faces in 16 ranges, finished Z rows "
                                "written to host memory while the next range is assembled)" if sym else
                                "mesh_MOM_3d.assemble_Z_rwg(out_host=...) (C ABI mb_mom_zmat_rwg_to_host_c64: "
                                "Z rows in 16 ranges, each range's D2H overlapping the next range's assembly)")
                               + ", pinned host buffers, H2D inputs + Z D2H inside the timed region"}
        del h_Z

    if rank == 0 and not args.no_cpu_baseline:
        wl = args.workload if not sym else args.workload.replace("sym", "ref")
        if wl in WORKLOADS:
            vals, info = cpu_sample_run(wl, args.cpu_seconds, steps=1)
            if sym:
                info["sample"] += " (the reference's own rule on the same mesh: the reference has no " \
                                  "symmetric-rule path)"
            line["cpu_baseline"] = {"value": vals[0], "unit": "pairs/s", **info}
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)


if __name__ == "__main__":
    main()
