#!/usr/bin/env python
"""Benchmark of the Helmholtz H-matrix BEM hot path on one GB300.

Headline workload (the large frequency sweep): pencil body -- cylinder of
radius 4 mm and length 0.2 m with a 10 mm conical tip and a flat back cap --
with exactly 81,920 flat triangles, Robin impedance walls (a = i k rho c / Z_e
with Z_e seeded log-uniform in [0.5, 50] rho c, b = 1), 8 right-hand sides
(g = 1 on the back-cap ring, and 7 seeded random-velocity patches on ~5 % of
the elements), 64 log-spaced frequencies 200 Hz - 8 kHz, c = 343 m/s,
rho = 1.2, leaf 32, eta = 2, ACA tol 1e-5, GMRES tol 1e-10 with the rank-2
H-LU preconditioner, Kirkup coupling.

A step is one frequency of that sweep solved completely for all 8
right-hand sides: near field, ACA assembly of both H-matrices, H-LU
factorization of the truncated system matrix (GPU task program), right-hand
sides, preconditioned GMRES inside FP64 iterative refinement, BC
back-substitution and pressure. The K timed steps are K of the 64
frequencies spread evenly over the band (all 64 when K >= 64); the W warm-up
solves use frequencies between them. Every step's working set (the
H-matrices and factors, GBs) is far larger than the 129 MB L2, so no explicit
flush is needed.

Two arms of the same method run on the GPU:
  mixed (headline) -- FP32 regular quadrature with FP64-formed centroid
      differences, FP64 singular/near-singular rules, complex-FP32 storage,
      FP32 H-LU factors (GPU task program), FP32-arithmetic inner GMRES inside
      FP64 iterative refinement, and the learned rule table for the ACA
      entries (--no-aca-rules: 16 points);
  plain            -- complex FP64 throughout (FP64 H-LU on the GPU too),
      timed on 2 of the K frequencies (the lowest and the highest).

  value : freq-solves/s with g resident in GPU memory (bem_solve_device)
  e2e   : freq-solves/s through bem_solve with host buffers (g copied in and
          p copied out inside the timed region, every step)

Legs riding along in the same line: the plain arm (``plain_fp64``), the
accuracy of the mixed arm against the FP64 oracle on the same body with 5,120
triangles (``accuracy_vs_oracle``), the 20,480-triangle pulsating sphere at
1.5 kHz (``sphere20k``: its own freq-solves/s, the plain arm and the oracle's
solve), the field at 20,480 observation points, the sphere above a rigid plane
and the 64-frequency box sweep; ``--no-plain``, ``--no-accuracy``,
``--no-sphere``, ``--no-field``, ``--no-half-space``, ``--no-sweep``,
``--no-cpu-baseline`` skip them. The CPU baseline is the oracle (FP64
C++/OpenMP restatement of the reference path, H-LU preconditioned) on all host
cores, one frequency of the headline workload.

``--impl reference`` times that CPU restatement alone on the headline
workload (full frequency solves within a time budget).
"""
from __future__ import annotations

import argparse
import importlib
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

FREQ = 1500.0
C0, RHO = 343.0, 1.2
ACA_TOL, GMRES_TOL = 1e-5, 1e-10
PENCIL_N, PENCIL_F = 81920, (200.0, 8000.0, 64)
WORKLOADS = {
    # name: (icosphere subdivisions, description)
    "sphere20k": (5, "pulsating sphere r=1 m, icosphere 20,480 triangles, f=1.5 kHz"),
    "sphere5k": (4, "pulsating sphere r=1 m, icosphere 5,120 triangles, f=1.5 kHz (profiling case)"),
}
PENCIL_DESC = ("pencil r=4 mm L=0.2 m + 10 mm conical tip, 81,920 triangles, impedance walls "
               "Z in [0.5, 50] rho c, 8 RHS, 64 log-spaced f 200 Hz-8 kHz, H-LU preconditioner "
               "rank 2")
# DRAM bytes per algorithmic byte of the 8-RHS FP32 H-matvec, measured with
# ncu (dram__bytes_read.sum + dram__bytes_write.sum of hmv_vpass<ArF32, 8> and
# hmv_upass<ArF32, 8>) on the 20,480-triangle pencil: 423 MB for 384 MB; the
# traffic grows with the stored entries, so it scales to the headline size
HMV32_R8_TRAFFIC_PER_BYTE = 422.9 / 384.0
# ncu of aca_kernel<0,float2,128,1> (the 128-thread ACA launch of the phi
# matrix) on the 20,480-triangle sphere at 1.5 kHz: FMA pipe active 37.8 % of
# its peak, issue slots 66 %, warps active 50 %, L2 hit rate 66 %
ACA_FMA_PIPE_NCU = 0.378
METRIC = "freq-solves/sec (H-matrix Helmholtz BEM solve, <=1e-5 rel. surface-pressure error)"
UNIT = "freq-solves/s"


def freqs(count, offset=0):
    """Distinct frequencies near 1.5 kHz (index i -> 1500 (1 + 1e-4 i))."""
    return [FREQ * (1.0 + 1e-4 * (offset + i)) for i in range(count)]


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx),
                "reasons": sorted(reasons), "samples": len(sm)}


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


def max_over_ranks(torch, value, ws, device="cuda"):
    """The slowest rank's time (replicas: every rank solves the same
    workload; the job takes as long as its slowest GPU)."""
    if ws <= 1:
        return float(value)
    t = torch.tensor([float(value)], device=device, dtype=torch.float64)
    torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    return float(t.item())


def matvec_bytes(info, ranks, n, elem, R=1):
    """Algorithmic bytes of one H-matvec: stored entries once (near-field
    m*n, low-rank (m+n)*k + k), plus each block's x segment and y once."""
    near = info[:, 4] == 0
    far = ~near
    m, nn = info[:, 1], info[:, 3]
    k = np.where(far, ranks, 0)
    mat = (m[near] * nn[near]).sum() * elem + ((m[far] + nn[far]) * k[far]).sum() * elem \
        + k[far].sum() * elem
    vec = R * (nn.sum() * 16 + 2 * n * 16)
    return int(mat + vec)


def make_solver(pkg, meshes, sub, precision, **extra):
    tri = meshes.icosphere(sub, 1.0)
    n = tri.shape[0]
    s = pkg.Solver(aca_tol=ACA_TOL, gmres_tol=GMRES_TOL, wave_speed=C0, density=RHO,
                   precision=precision, **extra)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    return s, n


def time_matvec(torch, pkg, s, n, reps=50, R=1):
    """Average duration of one system-matrix H-matvec of R vectors as the
    inner GMRES runs it (complex-FP32 storage, FP32 arithmetic: vector
    conversion, pass V, pass U), with CUDA events on the library's stream."""
    L = pkg.lib()
    stream = torch.cuda.ExternalStream(L.bem_stream(s._h))
    x = torch.randn(n * R, dtype=torch.complex128, device="cuda")
    y = torch.zeros(n * R, dtype=torch.complex128, device="cuda")
    for _ in range(3):
        L.bem_hmatvec_device_ex(s._h, 1, x.data_ptr(), y.data_ptr(), R, 0, pkg.BEM_ARITH_FP32)
    h0, h1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    h0.record(stream)
    for _ in range(reps):
        L.bem_hmatvec_device_ex(s._h, 1, x.data_ptr(), y.data_ptr(), R, 0, pkg.BEM_ARITH_FP32)
    h1.record(stream)
    torch.cuda.synchronize()
    return h0.elapsed_time(h1) / reps


def box_sweep(pkg, meshes, torch):
    """The batched sweep on the closed box with a piston: 5,120-triangle
    surface, 64 log-spaced frequencies 50-2000 Hz x 4 right-hand sides (piston
    + 3 random patches), mixed precision; sequential vs autotuned workers."""
    tri = meshes.box(n_target=5120, exact=True)
    n = tri.shape[0]
    g = meshes.box_piston_rhs(tri)
    freqs = meshes.log_frequencies(64, 50.0, 2000.0)
    out = {"workload": f"closed box 0.3x0.2x0.4 m, {n} triangles, piston r=0.05 m + 3 patches, "
                       "64 log-spaced f 50-2000 Hz", "nrhs": int(g.shape[1]), "freqs": 64}
    for name, workers in (("sequential", 1), ("batched", 0)):
        s = pkg.Solver(aca_tol=ACA_TOL, gmres_tol=GMRES_TOL, wave_speed=C0, density=RHO,
                       precision=1, sweep_workers=workers)
        s.set_mesh(tri)
        s.set_bc(np.zeros(n), np.ones(n))
        tune = None
        if workers == 0:
            t0 = time.perf_counter()
            tune = s.autotune(float(freqs[32]), g.shape[1])
            out["autotune_s"] = round(time.perf_counter() - t0, 3)
        s.sweep(freqs[:2], g)  # warm-up (allocations)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        p, info = s.sweep(freqs, g)
        dt = time.perf_counter() - t0
        out[name] = {"freq_solves_per_s": round(64 / dt, 3), "seconds": round(dt, 3),
                     "max_iterations": int(max(i["iterations"] for i in info)),
                     "all_converged": bool(all(i["status"] == 0 for i in info))}
        if tune:
            out[name]["tuned"] = tune
        if name == "sequential":
            p_seq = p
        else:
            out["rel_diff_batched_vs_sequential"] = float(np.linalg.norm(p - p_seq)
                                                          / np.linalg.norm(p_seq))
        s.close()
    return out


def field_eval(pkg, meshes, torch, s, n, sub, cpu=True, reps=10):
    """Field evaluation after the solve (bem_field; calculateFieldSolution,
    boundaryelementsolver.cpp:2192-2249): sound pressure at the 20,480
    triangle midpoints of a radius-2 m observation sphere from the mixed-
    precision boundary solution at 1.5 kHz. Kernel time with the data
    resident (bem_field_device, CUDA events on the library's stream), end to
    end through bem_field with host buffers, the analytic field
    p(r) = p(a) (a / r) exp(ik(r - a)) as accuracy check, and the oracle's
    dense FP64 sum on all host cores over a 256-point sample."""
    L = pkg.lib()
    tri = meshes.icosphere(sub, 1.0)
    obs = meshes.icosphere(5, 2.0)
    pts = np.ascontiguousarray((obs[:, 0:3] + obs[:, 3:6] + obs[:, 6:9]) / 3.0)
    M = pts.shape[0]
    phi, dphi, _, _ = s.solve(FREQ, np.ones(n))
    stream = torch.cuda.ExternalStream(L.bem_stream(s._h))
    dpts = torch.from_numpy(pts).to("cuda")
    dph = torch.from_numpy(phi[:, 0].copy()).to("cuda")
    ddph = torch.from_numpy(dphi[:, 0].copy()).to("cuda")
    dpf = torch.zeros(M, dtype=torch.complex128, device="cuda")
    dpp = torch.zeros(M, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()

    def run():
        s.field_device(FREQ, dpts.data_ptr(), M, dph.data_ptr(), ddph.data_ptr(), 1,
                       dpf.data_ptr(), dpp.data_ptr())
    for _ in range(3):
        run()
    torch.cuda.synchronize()
    l0 = s.launch_count()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(reps):
        run()
    e1.record(stream)
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / reps
    launches = (s.launch_count() - l0) // reps
    t0 = time.perf_counter()
    for _ in range(3):
        _, pp = s.field(FREQ, pts, phi[:, 0], dphi[:, 0])
    e2e_ms = (time.perf_counter() - t0) / 3 * 1e3
    k = 2 * np.pi * FREQ / C0
    pa = RHO * C0 * (1j * k) / (1j * k - 1)
    r = np.linalg.norm(pts, axis=1)
    ex = pa * (1.0 / r) * np.exp(1j * k * (r - 1.0))
    pairs = float(n) * M
    out = {
        "workload": f"{n}-element boundary solution -> {M} observation points "
                    "(midpoints of an r=2 m icosphere), 7-point rule, mixed precision",
        "kernel_ms": round(ms, 4), "launches_per_eval": int(launches),
        "gpairs_per_s": round(pairs / (ms * 1e-3) / 1e9, 2),
        "e2e_ms": round(e2e_ms, 3),
        "h2d_bytes": int(M * 24 + 2 * n * 16), "d2h_bytes": int(2 * M * 16),
        "analytic_rel_err": float(np.abs(pp[:, 0] - ex).max() / np.abs(ex).max()),
    }
    if cpu:
        import oracle
        sample = 256
        cores = os.cpu_count() or 1
        t0 = time.perf_counter()
        _, op = oracle.field(tri, FREQ, pts[:sample], phi[:, 0], dphi[:, 0], c=C0, rho=RHO,
                             nthreads=cores)
        cpu_s = (time.perf_counter() - t0) * M / sample
        out["rel_err_vs_oracle_sample"] = float(np.linalg.norm(pp[:sample, 0] - op[:, 0])
                                                / np.linalg.norm(op[:, 0]))
        out["cpu_oracle"] = {"s_per_eval": round(cpu_s, 3), "cores": cores, "kind": "port",
                             "sample": f"{sample} of {M} points, scaled"}
        out["speedup_vs_cpu_oracle"] = round(cpu_s / (e2e_ms * 1e-3), 1)
    return out


def half_space(pkg, meshes, torch, reps=3):
    """One impedance plane (bem_set_impedance_plane): the same sphere moved to
    1.2 m above the rigid plane z = 0 (gap 0.2 m), solved with and without the
    plane; mixed precision, the headline's tolerances."""
    tri = meshes.icosphere(WORKLOADS["sphere20k"][0], 1.0)
    tri[:, 2::3] += 1.2
    n = tri.shape[0]
    out = {"workload": f"pulsating sphere r=1 m, {n} triangles, centre 1.2 m above a rigid "
                       "plane, f=1.5 kHz"}
    p_by = {}
    for name, plane in (("free", False), ("plane", True)):
        s = pkg.Solver(aca_tol=ACA_TOL, gmres_tol=GMRES_TOL, wave_speed=C0, density=RHO,
                       precision=1, selector=2)
        s.set_mesh(tri)
        s.set_bc(np.zeros(n), np.ones(n))
        if plane:
            s.set_impedance_plane([0.0, 0.0, 0.0], [0.0, 0.0, 1.0])
        g = np.ones(n)
        for i in range(2):
            s.solve(FREQ * (1 + 1e-4 * i), g)
        best, info = None, None
        for i in range(reps):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            _, _, p, info = s.solve(FREQ * (1 + 1e-4 * (i + 2)), g)
            torch.cuda.synchronize()
            dt = time.perf_counter() - t0
            best = dt if best is None else min(best, dt)
        p_by[name] = p[:, 0]
        out[name] = {"ms_per_solve": round(best * 1e3, 2),
                     "t_aca_ms": round(info["t_aca"] * 1e3, 2),
                     "t_gmres_ms": round(info["t_gmres"] * 1e3, 2),
                     "gmres_iterations": int(info["iterations"]),
                     "max_rank": int(info["max_rank"]),
                     "capped_blocks": int(info["capped_blocks"])}
        s.close()
    out["rel_diff_plane_vs_free"] = float(np.linalg.norm(p_by["plane"] - p_by["free"])
                                          / np.linalg.norm(p_by["free"]))
    return out


def pencil_problem(meshes, n_target=PENCIL_N):
    """The pencil body, its 8 right-hand sides and wall admittances."""
    tri = meshes.pencil(n_target=n_target)
    return tri, meshes.pencil_rhs(tri), meshes.wall_admittance(tri.shape[0])


def pencil_solver(pkg, tri, beta, precision, **extra):
    extra.setdefault("aca_tol", ACA_TOL)
    extra.setdefault("sweep_workers", 1)
    s = pkg.Solver(gmres_tol=GMRES_TOL, wave_speed=C0, density=RHO,
                   precision=precision, use_preconditioner=1, precond_rank=2, gmres_maxit=1000,
                   **extra)
    s.set_mesh(tri)
    s.set_bc_impedance(beta)
    return s


def sweep_frequencies(meshes, steps, warmup):
    """K of the 64 log-spaced frequencies spread evenly over the band (all 64
    for K >= 64) and W warm-up frequencies at geometric midpoints of
    intervals spread over the band (none of them timed; the highest one
    first meets the largest ACA ranks, so any growth of the rank
    reservation happens before the timed region)."""
    f = meshes.log_frequencies(PENCIL_F[2], PENCIL_F[0], PENCIL_F[1])
    k = min(max(steps, 1), len(f))
    idx = np.unique(np.round(np.linspace(0, len(f) - 1, k)).astype(int))
    nw = min(max(warmup, 1), len(f) - 1)
    # the first warm-up lies 2 % above the band: its ACA ranks are the
    # largest, so the rank reservation grows there once (a new layout means a
    # new H-LU task program) and not inside the timed sweep
    wi = np.unique(np.round(np.linspace(len(f) - 2, 0, nw)).astype(int))[::-1]
    warm = [float(f[-1] * 1.02)] + [float(np.sqrt(f[i] * f[i + 1])) for i in wi[1:]]
    return [float(x) for x in f[idx]], warm


def timed_solves(torch, pkg, s, n, R, fr_timed, fr_warm, ws, g=None):
    """Warm-up solves, then the timed ones bracketed by barrier + sync, with
    the right-hand sides resident in GPU memory (bem_solve_device); per-step
    device times from events between the steps. Returns (ms, per-step ms,
    infos, p per step (steps x n x R), launches)."""
    stream = torch.cuda.ExternalStream(pkg.lib().bem_stream(s._h))
    if g is None:
        g = torch.ones(n * R, dtype=torch.complex128, device="cuda")
    p = torch.zeros((len(fr_timed), R, n), dtype=torch.complex128, device="cuda")
    for f in fr_warm:
        s.solve_device(f, g.data_ptr(), R, 0, 0, p[0].data_ptr())
    torch.cuda.synchronize()
    if ws > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    l0 = s.launch_count()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(len(fr_timed) + 1)]
    infos = []
    ev[0].record(stream)
    for i, f in enumerate(fr_timed):
        infos.append(s.solve_device(f, g.data_ptr(), R, 0, 0, p[i].data_ptr()))
        ev[i + 1].record(stream)
    torch.cuda.synchronize()
    if ws > 1:
        torch.distributed.barrier()
    ms = max_over_ranks(torch, ev[0].elapsed_time(ev[-1]), ws)
    per = [ev[i].elapsed_time(ev[i + 1]) for i in range(len(fr_timed))]
    pn = p.cpu().numpy().transpose(0, 2, 1)  # steps x n x R
    return ms, per, infos, pn, s.launch_count() - l0


def rel_err_cols(p, ref):
    """Largest relative 2-norm difference over the columns (right-hand sides)."""
    return float(max(np.linalg.norm(p[:, r] - ref[:, r]) / np.linalg.norm(ref[:, r])
                     for r in range(ref.shape[1])))


def accuracy_vs_oracle(pkg, meshes, n_target=5120, fr=(200.0, 1000.0, 8000.0)):
    """The GPU arms against the FP64 oracle (H-LU preconditioned, all host
    cores) on the same pencil body with 5,120 triangles: the oracle at the
    workload's tolerances (the same approximation) and at ACA 1e-7 / GMRES
    1e-12 (the converged reference). Arms: the headline's mixed arm, the
    same with the FP64 near field in the refinement residual, the latter at
    ACA 1e-6, and the plain complex-FP64 arm."""
    import oracle
    tri, g, beta = pencil_problem(meshes, n_target)
    n = tri.shape[0]
    cores = os.cpu_count() or 1
    P = oracle.Problem(tri, 32, 2.0)
    out = {"workload": f"pencil as the headline with {n} triangles, 8 RHS, f = "
                       + ", ".join(f"{f:g}" for f in fr) + " Hz"}
    arms = {}
    for name, prec, extra in (("mixed", 1, {"selector": 2}),
                              ("mixed_fp64_near", 1, {"selector": 2, "near_fp64": 1}),
                              ("mixed_aca1e-6_fp64_near", 1, {"near_fp64": 1, "aca_tol": 1e-6}),
                              ("plain", 0, {})):
        s = pencil_solver(pkg, tri, beta, prec, **extra)
        arms[name] = [s.solve(f, g, want=("p",))[2] for f in fr]
        s.close()
    t0 = time.perf_counter()
    refs = {}
    for key, aca, gt in (("same_tol", ACA_TOL, GMRES_TOL), ("aca1e-7", 1e-7, 1e-12)):
        refs[key] = []
        for f in fr:
            k = 2 * np.pi * f / C0
            _, _, p, _ = P.solve(f, C0, RHO, 2, 1j * k * beta, np.ones(n), g, aca, gt,
                                 nthreads=cores, precond_rank=2)
            refs[key].append(p)
    out["oracle_s"] = round(time.perf_counter() - t0, 2)
    for name, ps in arms.items():
        for key, rs in refs.items():
            out[f"{name}_vs_oracle_{key}"] = max(rel_err_cols(a, b) for a, b in zip(ps, rs))
    return out


def sphere_leg(torch, pkg, meshes, args, ws):
    """The 20,480-triangle pulsating sphere at 1.5 kHz (ACA 1e-5, GMRES 1e-10,
    no preconditioner, as the reference's default): mixed freq-solves/s, the
    plain arm, the oracle's solve of the same workload and the errors of the
    GPU arms against it, the field, the half-space and the box sweep legs."""
    sub = WORKLOADS["sphere20k"][0]
    steps = max(1, min(args.steps, 8))
    fr_t = freqs(steps, 0)
    fr_w = freqs(args.warmup, -args.warmup - 1)
    out = {"workload": WORKLOADS["sphere20k"][1] + ", ACA 1e-5, GMRES 1e-10, 1 RHS"}
    s, n = make_solver(pkg, meshes, sub, 1, selector=0 if args.no_aca_rules else 2)
    ms, _, infos, pm, _ = timed_solves(torch, pkg, s, n, 1, fr_t, fr_w, ws)
    out["mixed"] = {"freq_solves_per_s": round(steps / (ms / 1e3), 3),
                    "ms_per_solve": round(ms / steps, 3),
                    "gmres_iterations": int(max(i["iterations"] for i in infos))}
    # the ACA phase of the last timed solve: entries evaluated per second
    # (k (m + n) per block of rank k, both matrices) and the FMA-pipe share
    part = s.partition()
    E = aca_entries(part, s.ranks(0)) + aca_entries(part, s.ranks(1))
    t_aca = infos[-1]["t_aca"]
    out["aca"] = {"frequency_hz": fr_t[-1], "span_ms": round(1e3 * t_aca, 3), "entries": E,
                  "entries_per_s": round(E / t_aca), "bound": "issue / FP32 pipes",
                  "fma_pipe_active_ncu": ACA_FMA_PIPE_NCU,
                  "fma_pipe_source": "ncu --set full of aca_kernel<0,float2,128>, this "
                                     "workload at 1.5 kHz"}
    if not args.no_plain:
        s64, _ = make_solver(pkg, meshes, sub, 0)
        ms64, _, _, p64, _ = timed_solves(torch, pkg, s64, n, 1, fr_t[:2], fr_w[:1], ws)
        s64.close()
        out["plain_fp64"] = {"freq_solves_per_s": round(2 / (ms64 / 1e3), 3),
                             "ms_per_solve": round(ms64 / 2, 2)}
        out["rel_err_mixed_vs_plain"] = max(rel_err_cols(pm[i], p64[i]) for i in range(2))
    k = 2 * np.pi * fr_t[-1] / C0
    pa = RHO * C0 * (1j * k) / (1j * k - 1)
    out["analytic_rel_err"] = round(float(np.abs(pm[-1] - pa).max() / abs(pa)), 5)
    if not args.no_cpu_baseline:
        import oracle
        tri = meshes.icosphere(sub, 1.0)
        cores = os.cpu_count() or 1
        t0 = time.perf_counter()
        _, _, po, st = oracle.Problem(tri, 32, 2.0).solve(
            fr_t[-1], C0, RHO, 2, np.zeros(n), np.ones(n), np.ones(n), ACA_TOL, GMRES_TOL,
            nthreads=cores)
        dt = time.perf_counter() - t0
        out["cpu_oracle"] = {"freq_solves_per_s": round(1.0 / dt, 5), "cores": cores,
                             "kind": "port", "gmres_iterations": int(st["iters"])}
        out["rel_err_mixed_vs_oracle"] = rel_err_cols(pm[-1], po)
        if "plain_fp64" in out:
            s64, _ = make_solver(pkg, meshes, sub, 0)
            _, _, p64l, _ = s64.solve(fr_t[-1], np.ones(n), want=("p",))
            s64.close()
            out["rel_err_plain_vs_oracle"] = rel_err_cols(p64l, po)
    if not args.no_field:
        out["field_eval"] = field_eval(pkg, meshes, torch, s, n, sub, cpu=not args.no_cpu_baseline)
    s.close()
    if not args.no_half_space:
        out["half_space"] = half_space(pkg, meshes, torch)
    if not args.no_sweep:
        out["box_sweep"] = box_sweep(pkg, meshes, torch)
    return out


def cpu_pencil_solve(f, nthreads, n_target=PENCIL_N):
    """One frequency of the headline workload on the host cores with the
    oracle (FP64, H-LU preconditioned GMRES, 8 right-hand sides)."""
    import oracle
    meshes = importlib.import_module("3d_bem_gb300.meshes")
    oracle.build()
    tri, g, beta = pencil_problem(meshes, n_target)
    n = tri.shape[0]
    P = oracle.Problem(tri, 32, 2.0)
    k = 2 * np.pi * f / C0
    t0 = time.perf_counter()
    _, _, p, st = P.solve(f, C0, RHO, 2, 1j * k * beta, np.ones(n), g, ACA_TOL, GMRES_TOL,
                          nthreads=nthreads, precond_rank=2, maxit=1000)
    return time.perf_counter() - t0, st, p


def run_ours(args):
    import torch
    ws, rank, local = dist_env()
    if ws > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")
    torch.cuda.set_device(local)
    pkg = importlib.import_module("3d_bem_gb300")
    meshes = importlib.import_module("3d_bem_gb300.meshes")
    pkg.build()
    tri, g_host, beta = pencil_problem(meshes)
    n, R = tri.shape[0], g_host.shape[1]
    fr_t, fr_w = sweep_frequencies(meshes, args.steps, max(args.warmup, 1))
    g_dev = torch.from_numpy(np.ascontiguousarray(g_host.T)).reshape(-1).to("cuda")
    learned = (1 if args.selector else 0) | (0 if args.no_aca_rules else 2)
    extra = {"selector": learned} if learned else {}
    extra["near_fp64"] = 1 if args.near_fp64 else 0

    # batched sweep: W concurrent frequency workers (each its own stream,
    # buffers and H-LU factors), K frequencies; g and p resident in GPU memory
    W = max(1, args.workers)
    s = pencil_solver(pkg, tri, beta, 1, sweep_workers=W, **extra)
    p_dev = torch.zeros((len(fr_t), R, n), dtype=torch.complex128, device="cuda")
    stream = torch.cuda.ExternalStream(pkg.lib().bem_stream(s._h))
    # warm-up: one solve plans the H-LU task program (the workers inherit
    # it), then a sweep with every worker busy
    warm = [fr_w[i % len(fr_w)] * (1.0 + 1e-3 * i) for i in range(max(W, len(fr_w)))]
    p_warm = torch.zeros((len(warm), R, n), dtype=torch.complex128, device="cuda")
    s.solve_device(warm[0], g_dev.data_ptr(), R, 0, 0, p_warm[0].data_ptr())
    s.sweep_device(warm, g_dev.data_ptr(), R, p_warm.data_ptr())
    torch.cuda.synchronize()
    if ws > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    clk = Clocks(local)
    clk.start()
    l0 = s.launch_count()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    infos = s.sweep_device(fr_t, g_dev.data_ptr(), R, p_dev.data_ptr())
    e1.record(stream)
    torch.cuda.synchronize()
    clocks = clk.stop()
    launches = s.launch_count() - l0  # the first handle's own kernels
    if ws > 1:
        torch.distributed.barrier()
    ms = max_over_ranks(torch, e0.elapsed_time(e1), ws)
    pm = p_dev.cpu().numpy().transpose(0, 2, 1)  # steps x n x R
    K = len(fr_t)
    value = ws * K / (ms / 1e3)
    per = [1e3 * i["t_total"] for i in infos]

    # end to end through bem_sweep: pinned host g in, host p out (every
    # frequency's pressures copied back), the same workers
    gh = torch.from_numpy(np.ascontiguousarray(g_host.T)).pin_memory()
    gpin = gh.numpy().T
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    s.sweep(fr_t, gpin)
    torch.cuda.synchronize()
    e2e = ws * K / (time.perf_counter() - t0)

    # roofline of the inner-GMRES H-matvec (complex-FP32 storage, FP32
    # arithmetic, the 8 right-hand sides of a product; matrix bytes read once)
    info_part = s.partition()
    ranks = s.ranks(1)
    B = matvec_bytes(info_part, ranks, n, elem=8, R=R)
    mv_ms = time_matvec(torch, pkg, s, n, R=R)
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except (OSError, ValueError):
        pass
    hbm = float(peaks.get("hbm_gbs", 6800.0))
    achieved = B / (mv_ms * 1e-3) / 1e9
    phase = {key: round(float(np.mean([i[key] for i in infos])), 5)
             for key in ("t_nearfield", "t_aca", "t_rhs", "t_precond", "t_gmres", "t_total")}
    line = {
        "metric": METRIC, "value": round(value, 4), "unit": UNIT, "n_gpus": ws,
        "steps": K, "warmup": len(fr_w), "ms_per_step": round(ms / K, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "c64 storage + fp32 quadrature/H-LU, fp64 refinement/Arnoldi/singular rules",
        "data": "synthetic (seeded pencil mesh, wall impedances and velocity patches)",
        "config": {"workload": PENCIL_DESC, "n_elements": n, "nrhs": R,
                   "frequencies_timed_hz": [round(f, 2) for f in fr_t],
                   "aca_tol": ACA_TOL, "gmres_tol": GMRES_TOL, "leaf_size": 32, "eta": 2.0,
                   "coupling": "Kirkup", "bc": "Robin impedance walls a = i k rho c / Z",
                   "precision": "mixed", "hlu_preconditioner": "rank 2, factorized on the GPU",
                   "batching": f"{W} concurrent frequency workers x 8 RHS (bem_sweep_device)",
                   "learned_selector": bool(args.selector),
                   "learned_aca_rules": not args.no_aca_rules,
                   "near_field": "complex FP32 in GMRES; FP64 (two complex-FP32 parts) in the "
                                 "refinement residual" if args.near_fp64 else "complex FP32",
                   "parallelism": f"replicas{ws}" if ws > 1 else "single-gpu",
                   "l2": "working set (H-matrices and factors, GBs) >> 129 MB L2; no flush"},
        "e2e": {"value": round(e2e, 4), "unit": UNIT, "h2d_bytes_per_step": n * R * 16,
                "d2h_bytes_per_step": n * R * 16},
        "roofline": {"kernel": "hmatvec FP32 (hmv_vpass + hmv_upass), c64 storage, 8 RHS",
                     "bound": "hbm", "achieved": round(achieved, 1), "peak": hbm, "unit": "GB/s",
                     "frac": round(achieved / hbm, 4),
                     "traffic": int(B * HMV32_R8_TRAFFIC_PER_BYTE),
                     "traffic_source": "ncu DRAM bytes per algorithmic byte on the 20,480-"
                                       "triangle pencil, scaled by the algorithmic bytes",
                     "bytes_per_launch": B, "ms_per_launch": round(mv_ms, 4),
                     "peak_source": "MEASURED_PEAKS.json hbm_gbs" if peaks else "fallback"},
        "gpu_launches": int(launches),
        "phases_s": phase,
        "worker_ms_per_frequency": [round(x, 1) for x in per],
        "gmres_iterations": int(max(i["iterations"] for i in infos)),
        "true_residual": float(max(i["true_residual"] for i in infos)),
        "all_converged": bool(all(i["status"] == 0 for i in infos)),
        "max_rank": int(max(i["max_rank"] for i in infos)),
        "clocks": clocks,
    }
    s.close()
    if not args.no_plain and ws == 1:
        # the plain method: complex FP64 throughout, one frequency after the
        # other (no concurrent workers), at the lowest, middle and highest
        # timed frequencies (its cost per frequency falls with frequency, as
        # the GMRES step counts do)
        s64 = pencil_solver(pkg, tri, beta, 0)
        pick = sorted({fr_t[0], fr_t[len(fr_t) // 2], fr_t[-1]})
        ms64, per64, i64, p64, _ = timed_solves(torch, pkg, s64, n, R, pick, fr_w[:1], ws, g_dev)
        s64.close()
        line["plain_fp64"] = {
            "frequencies_hz": [round(f, 2) for f in pick],
            "ms_per_frequency": [round(x, 1) for x in per64],
            "mean_ms_per_frequency": round(float(np.mean(per64)), 1),
            "mixed_sweep_ms_per_frequency": round(ms / K, 1),
            "speedup_mixed_vs_plain": round(float(np.mean(per64)) / (ms / K), 2),
            "phases_s": {key: round(float(np.mean([i[key] for i in i64])), 4)
                         for key in ("t_nearfield", "t_aca", "t_precond", "t_gmres", "t_total")},
            "rel_err_mixed_vs_plain": max(rel_err_cols(pm[fr_t.index(f)], p64[j])
                                          for j, f in enumerate(pick))}
    if not args.no_accuracy and ws == 1:
        line["accuracy_vs_oracle"] = accuracy_vs_oracle(pkg, meshes)
    if not args.no_sphere and ws == 1:
        line["sphere20k"] = sphere_leg(torch, pkg, meshes, args, ws)
    if not args.no_cpu_baseline and rank == 0 and ws == 1:
        cores = os.cpu_count() or 1
        f = fr_t[len(fr_t) // 2]
        dt, st, po = cpu_pencil_solve(f, cores)
        line["rel_err_mixed_vs_oracle"] = {"frequency_hz": round(f, 2),
                                           "value": rel_err_cols(pm[fr_t.index(f)], po)}
        line["cpu_baseline"] = {"value": round(1.0 / dt, 5), "unit": UNIT, "cores": cores,
                                "kind": "port",
                                "sample": f"one frequency ({f:.0f} Hz) of the workload, 8 RHS, "
                                          f"{dt:.1f} s (assembly, H-LU {st['t_factor']:.1f} s, "
                                          f"GMRES {int(st['iters'])} iterations)"}
    if rank == 0:
        print(json.dumps(line), flush=True)
    if ws > 1:
        torch.distributed.destroy_process_group()


def run_hlu_only(args):
    """One H-LU factorization of the pencil on the GPU, after a warm-up one
    (for profiling the executor kernel): mixed precision, rank 2, 1 kHz,
    args.pencil_n triangles."""
    import torch
    pkg = importlib.import_module("3d_bem_gb300")
    meshes = importlib.import_module("3d_bem_gb300.meshes")
    pkg.build()
    tri, _, beta = pencil_problem(meshes, args.pencil_n)
    s = pencil_solver(pkg, tri, beta, 1, selector=2, near_fp64=1)
    s.assemble(1000.0)
    s.hlu_build()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    s.hlu_build()
    torch.cuda.synchronize()
    print(json.dumps({"hlu_only": {"n_elements": int(tri.shape[0]),
                                   "seconds": round(time.perf_counter() - t0, 4)}}), flush=True)
    s.close()


def run_hmatvec_only(args):
    """The inner-GMRES H-matvec of the pencil (complex-FP32 storage, FP32
    arithmetic, 8 right-hand sides) after one assembly at 1 kHz, args.pencil_n
    triangles: its algorithmic bytes and event-timed duration (for profiling
    the hmv_vpass and hmv_upass kernels)."""
    import torch
    pkg = importlib.import_module("3d_bem_gb300")
    meshes = importlib.import_module("3d_bem_gb300.meshes")
    pkg.build()
    tri, g, beta = pencil_problem(meshes, args.pencil_n)
    n, R = tri.shape[0], g.shape[1]
    s = pencil_solver(pkg, tri, beta, 1, selector=2)
    s.assemble(1000.0)
    B = matvec_bytes(s.partition(), s.ranks(1), n, elem=8, R=R)
    ms = time_matvec(torch, pkg, s, n, reps=10, R=R)
    print(json.dumps({"hmatvec_only": {"n_elements": int(n), "nrhs": R, "bytes": int(B),
                                       "ms": round(ms, 4),
                                       "gbs": round(B / (ms * 1e-3) / 1e9, 1)}}), flush=True)
    s.close()


def aca_entries(partition, ranks):
    """ACA entries of one matrix: a block of rank k (m x n) evaluates k rows and
    k columns of itself, k (m + n) entries (the rejected last step not counted)."""
    adm = partition[:, 4] != 0
    m, n = partition[adm, 1], partition[adm, 3]
    return int(np.sum(ranks[adm].astype(np.int64) * (m + n)))


def run_aca_only(args):
    """Assembly of the 20,480-triangle sphere at 1.5 kHz (mixed precision, ACA
    1e-5, the learned ACA rule table), a warm-up one and three timed ones: the
    ACA span and its entries per second (for profiling aca_kernel)."""
    import torch
    pkg = importlib.import_module("3d_bem_gb300")
    meshes = importlib.import_module("3d_bem_gb300.meshes")
    pkg.build()
    s, n = make_solver(pkg, meshes, WORKLOADS["sphere20k"][0], 1, selector=2)
    s.assemble(1500.0)
    torch.cuda.synchronize()
    ts = []
    for _ in range(3):
        t0 = time.perf_counter()
        s.assemble(1500.0)
        torch.cuda.synchronize()
        ts.append(time.perf_counter() - t0)
    part = s.partition()
    E = aca_entries(part, s.ranks(0)) + aca_entries(part, s.ranks(1))
    t = min(ts)
    print(json.dumps({"aca_only": {"n_elements": int(n), "assemble_ms": round(1e3 * t, 3),
                                   "aca_entries": E,
                                   "entries_per_s": round(E / t, 1)}}), flush=True)
    s.close()


def run_field_only(args):
    """The field leg alone on one GPU (for profiling its kernels)."""
    import torch
    pkg = importlib.import_module("3d_bem_gb300")
    meshes = importlib.import_module("3d_bem_gb300.meshes")
    pkg.build()
    sub = WORKLOADS[args.workload][0]
    s, n = make_solver(pkg, meshes, sub, 1)
    out = field_eval(pkg, meshes, torch, s, n, sub, cpu=not args.no_cpu_baseline)
    print(json.dumps({"field_eval": out}), flush=True)
    s.close()


def run_reference(args):
    """The oracle (the reference path restated on the CPU: FP64, H-LU
    preconditioned GMRES, all host cores) on the headline workload: each step
    one full frequency solve with 8 right-hand sides; warm-up and steps stop
    once the next solve would pass the time budget (the counts are reported)."""
    ws, rank, local = dist_env()
    if rank != 0:
        return
    meshes = importlib.import_module("3d_bem_gb300.meshes")
    cores = os.cpu_count() or 1
    budget = float(os.environ.get("BEM_REF_BUDGET_S", "300"))
    fr_t, fr_w = sweep_frequencies(meshes, args.steps, max(args.warmup, 1))
    t_start = time.perf_counter()
    warm = 0
    for f in fr_w:
        dt, _, _ = cpu_pencil_solve(f, cores)
        warm += 1
        if time.perf_counter() - t_start + 2 * dt > budget:
            break
    times, iters = [], []
    for f in fr_t:
        dt, st, _ = cpu_pencil_solve(f, cores)
        times.append(dt)
        iters.append(int(st["iters"]))
        if time.perf_counter() - t_start + dt > budget:
            break
    value = len(times) / sum(times)
    line = {
        "metric": METRIC, "value": round(value, 5), "unit": UNIT, "n_gpus": ws,
        "steps": len(times), "warmup": warm,
        "ms_per_step": round(1e3 * sum(times) / len(times), 1),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "c128 (fp64)", "data": "synthetic (seeded pencil mesh)",
        "config": {"workload": PENCIL_DESC, "n_elements": PENCIL_N, "nrhs": 8,
                   "frequencies_timed_hz": [round(f, 2) for f in fr_t[:len(times)]],
                   "aca_tol": ACA_TOL, "gmres_tol": GMRES_TOL, "leaf_size": 32, "eta": 2.0,
                   "coupling": "Kirkup", "precision": "fp64",
                   "hlu_preconditioner": "rank 2 (host)", "parallelism": "cpu-openmp"},
        "impl": "reference",
        "cpu_baseline": {"value": round(value, 5), "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{len(times)} full frequency solve(s) of the workload "
                                   f"(GMRES iterations {iters}); the reference itself needs Qt 6 "
                                   "+ Eigen and cannot be built here, so its CPU path is the "
                                   "oracle restatement"},
        "e2e": {"value": round(value, 5), "unit": UNIT, "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=16,
                    help="frequencies of the 64-frequency sweep timed (spread over the band)")
    ap.add_argument("--workers", type=int, default=8,
                    help="concurrent frequency workers of the batched sweep (mixed arm; eight "
                         "measured 2.70 freq-solves/s, six 2.45 on the same GPU, one 0.8-1.1)")
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="sphere20k", choices=sorted(WORKLOADS),
                    help="workload of --field-only")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-plain", action="store_true", help="skip the complex-FP64 arms")
    ap.add_argument("--no-accuracy", action="store_true",
                    help="skip the accuracy leg against the oracle (5,120-triangle pencil)")
    ap.add_argument("--no-sphere", action="store_true",
                    help="skip the 20,480-triangle sphere leg (and its field, half-space and "
                         "box-sweep legs)")
    ap.add_argument("--no-field", action="store_true",
                    help="skip the field evaluation at 20,480 observation points")
    ap.add_argument("--no-half-space", action="store_true",
                    help="skip the sphere-above-a-rigid-plane solves")
    ap.add_argument("--hlu-only", action="store_true",
                    help="only one H-LU factorization of the pencil (after a warm-up one); "
                         "profiling")
    ap.add_argument("--hmatvec-only", action="store_true",
                    help="only the pencil's inner-GMRES H-matvec (8 RHS); profiling")
    ap.add_argument("--pencil-n", type=int, default=PENCIL_N,
                    help="triangles of the pencil for --hlu-only / --hmatvec-only")
    ap.add_argument("--aca-only", action="store_true",
                    help="only assemblies of the 20,480-triangle sphere (ACA span, entries/s); "
                         "profiling")
    ap.add_argument("--field-only", action="store_true",
                    help="only the field evaluation leg (one mixed solve first); profiling")
    ap.add_argument("--no-sweep", action="store_true",
                    help="skip the batched box sweep (64 frequencies x 4 RHS)")
    ap.add_argument("--selector", action="store_true",
                    help="mixed arm: learned quadrature order per near-field pair")
    ap.add_argument("--near-fp64", action="store_true",
                    help="mixed arm: the refinement residual reads the near field in FP64 (two "
                         "complex-FP32 parts); on this body the difference to the FP64 arm is "
                         "the ACA approximation's, so it is off by default")
    ap.add_argument("--no-aca-rules", action="store_true",
                    help="mixed arm: the 16-point rule for the ACA entries instead of the "
                         "learned rule table")
    args = ap.parse_args()
    if args.hlu_only:
        run_hlu_only(args)
    elif args.hmatvec_only:
        run_hmatvec_only(args)
    elif args.field_only:
        run_field_only(args)
    elif args.aca_only:
        run_aca_only(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
