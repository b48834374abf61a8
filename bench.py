#!/usr/bin/env python
"""Benchmark: PCG solve time at 3.24M DOF (128x128x64 voxel block, 6 tets per
voxel, per-tet E log-uniform in [0.1, 10]), FP32-inner / FP64-refinement ILU(0)
PCG to |b - K u| / |b| < 1e-10, next to the plain FP64 GPU Solve_PCG and the
reference's CPU Solve_PCG.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

One step = one solve of K u = b from b resident in HBM (value), or through the
C ABI with host buffers (e2e). Prints one JSON line (rank 0).
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "PCG solve ms @3.2M DOF: FP32+FP64-refine vs FP64 to 1e-10; adjoint/forward"
WORKLOAD = dict(nx=128, ny=128, nz=64, h=1.0 / 128, e_lo=0.1, e_hi=10.0, seed=3, nu=0.3, rho=1.0,
                g=(0.0, 0.0, -1e-3), tol=1e-10, inner_tol=1e-4, refresh=0.1)
SMALL = dict(WORKLOAD, nx=32, ny=32, nz=16, h=1.0 / 32)
METHOD, OTHER = "reliable", "restart"  # refinement scheme of the headline solve / of the comparison
FALLBACK_HBM_GBS = 6800.0
# implicit cloth: 256x256-vertex sheet, E = 1e3, nu = 0.3, bending 1e-3, two corners pinned, dt = 0.01,
# ILU(0)-PCG to 1e-8 capped at the reference step's own 100 iterations, checkpoints every 10 steps
CLOTH = dict(ndiv=255, young=1e3, nu=0.3, stiff_bend=1e-3, g=(0.0, 0.0, -10.0), dt=0.01, tol=1e-8, max_iter=100,
             nsteps=100, ckpt_every=10, target_seed=5, target_sigma=0.01)
# the same cloth on the largest sheet whose ILU(0)-PCG still converges to 1e-8 (52x52 cells; at 56 cells the
# preconditioner already amplifies by 2e4, at 64 by 1e20), with no iteration cap
CLOTH_CONVERGING = dict(CLOTH, ndiv=52, max_iter=5000)


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


# ---------------------------------------------------------------------------
class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        os.unlink(self.path)
        if not rows:
            return None

        def num(x):
            try:
                return float(x)
            except ValueError:
                return float("nan")

        sm = [num(r[1]) for r in rows]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower() == "active"})
        return {"sm_mhz": float(np.nanmedian(sm)), "sm_max_mhz": float(np.nanmax([num(r[2]) for r in rows])),
                "reasons": reasons, "samples": len(rows),
                "power_w_max": float(np.nanmax([num(r[3]) for r in rows]))}


# ---------------------------------------------------------------------------
def algorithmic_bytes(kind: str, nb: int, nz: int, s: int) -> float:
    """Bytes one launch of a kernel class must move (each array once per pass).

    nb block rows, nz off-diagonal blocks, s = bytes per value; index arrays u32.
    nz/2 blocks lie in each triangle (the pattern is symmetric)."""
    v3 = 3 * s * nb
    if kind == "spmv":      # K values + col + row_start, p read, Ap written
        return 9 * s * (nz + nb) + 4 * nz + 4 * (nb + 1) + 2 * v3
    if kind == "fwd":       # L blocks + D^-1 + col/row_start/dia_ind/order, in read, out written
        return 9 * s * (nz / 2 + nb) + 4 * nz / 2 + 4 * (3 * nb + 1) + 2 * v3
    if kind == "bwd":       # U' blocks + col/row_start/dia_ind/order, in read, out written
        return 9 * s * (nz / 2) + 4 * nz / 2 + 4 * (3 * nb + 1) + 2 * v3
    if kind == "update":    # r, x, p, Ap read; r, x and the sweeps' two pending-marker outputs written
        return 8 * v3
    if kind == "dot":       # r, z read
        return 2 * v3
    if kind == "pupdate":   # p, z read; p written
        return 3 * v3
    return float("nan")


def traffic_from_profiles(kind: str):
    """DRAM bytes per launch recorded from an ncu capture (profiles/ncu_traffic.json)."""
    try:
        with open(os.path.join(ROOT, "profiles", "ncu_traffic.json")) as f:
            t = json.load(f)
        return t.get(kind)
    except Exception:
        return None


# ---------------------------------------------------------------------------
def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as dist
        import torch
        backend = "nccl" if torch.cuda.is_available() else "gloo"
        dist.init_process_group(backend=backend)
    return world, rank, local, dist


def reduce_max(dist, value: float, device=None) -> float:
    if dist is None:
        return value
    import torch
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def build_problem(w):
    import delfem2_gb300 as D
    t0 = time.perf_counter()
    arrays = D.voxel_problem_arrays(w["nx"], w["ny"], w["nz"], w["h"], seed=w["seed"],
                                    e_range=(w["e_lo"], w["e_hi"]))
    t1 = time.perf_counter()
    P = D.StaticElasticProblem(arrays, nu=w["nu"], rho=w["rho"], g=w["g"])
    t2 = time.perf_counter()
    return P, arrays, {"host_mesh_pattern_s": t1 - t0, "device_pattern_levels_s": t2 - t1}


def iterations_to(hist, tol):
    h = np.asarray(hist)
    k = np.nonzero(h / h[0] < tol)[0]
    return int(k[0]) if k.size else len(h) - 1


def cpu_port_ms_per_iter(P, b_host, iters: int):
    """Time `iters` Solve_PCG iterations of the C port on the device-assembled system."""
    from oracle import port
    O = port()
    a = P.a
    vc, vd = P.K.get_values()
    col, dia = P.ilu.pattern()
    ivc, ivd = P.ilu.values()
    O.solve_pcg(a["psup_ind"], a["psup"], vc, vd, col, dia, ivc, ivd, b_host, 1e-300, 1)  # warm-up
    t = time.perf_counter()
    O.solve_pcg(a["psup_ind"], a["psup"], vc, vd, col, dia, ivc, ivd, b_host, 1e-300, iters)
    return (time.perf_counter() - t) * 1e3 / iters


def cpu_full_solve_cfg2(iters_sample: int):
    """The reference's FP64 Solve_PCG (C restatement, one core) on the 64^3 voxel block (823,875 DOF, per-tet E
    log-uniform [0.1, 10], seed 2) timed to 1e-10 without scaling, next to the time projected from an
    `iters_sample`-iteration sample on the same system: the check that the headline's CPU figure (a sample scaled
    to the full iteration count) scales linearly."""
    import delfem2_gb300 as D
    from oracle import port
    O = port()
    a = D.voxel_problem_arrays(64, 64, 64, 1.0 / 64, seed=2, e_range=(0.1, 10.0))
    ind, psup = a["psup_ind"], a["psup"]
    np_ = a["np"]
    vc, vd, b = np.zeros(psup.size * 9), np.zeros(np_ * 9), np.zeros(np_ * 3)
    O.assemble_tet_linear(ind, psup, vc, vd, b, a["xyz"], a["tet"], a["young"], 0.3, 1.0, [0.0, 0.0, -1e-3])
    O.set_fixed_bc(ind, psup, vc, vd, a["bc"])
    O.rhs_zero(b, a["bc"])
    col, dia = O.ilu_pattern0(ind, psup)
    ivc, ivd = O.ilu_copy_value(ind, col, psup, vc, vd)
    O.ilu_decompose(ind, col, dia, ivc, ivd)
    O.solve_pcg(ind, psup, vc, vd, col, dia, ivc, ivd, b, 1e-300, 1)  # warm-up, as the headline's sample
    t = time.perf_counter()
    O.solve_pcg(ind, psup, vc, vd, col, dia, ivc, ivd, b, 1e-300, iters_sample)
    per = (time.perf_counter() - t) * 1e3 / iters_sample
    t = time.perf_counter()
    _, _, h = O.solve_pcg(ind, psup, vc, vd, col, dia, ivc, ivd, b, 1e-10, 100000)
    full_ms = (time.perf_counter() - t) * 1e3
    its = len(h) - 1
    return {"workload": f"64x64x64 voxels x 6 tets, {np_ * 3} DOF, FP64 ILU(0)-PCG to 1e-10 (C restatement, 1 core)",
            "iterations": its, "timed_ms": round(full_ms, 1), "projected_ms": round(per * its, 1),
            "projected_over_timed": round(per * its / full_ms, 3),
            "sample": f"{iters_sample} iterations at {per:.1f} ms each, scaled to {its}"}


def cloth_bench(dev, nsteps: int, cpu: bool, c=None):
    """The implicit-cloth workload: backward-Euler steps of StepTime_InternalDynamicsILU on the 256x256-vertex
    sheet (FP64 ILU(0)-PCG to 1e-8, at most 100 iterations per step as the reference's step caps it: ILU(0) of
    this system is unstable at this size, so PCG does not reach the tolerance), checkpoints every 10 steps, then
    the reverse pass for dL/dE_t of L = |x_N - x*|^2 / 2 with a seeded target x*. With `c` =
    CLOTH_CONVERGING, the same on the largest sheet where the solves converge."""
    import torch
    from delfem2_gb300 import cloth as DC
    c = c or CLOTH
    xyz0, _, tri, quad = DC.SetClothShape_Square(c["ndiv"], 1.0)
    cl = DC.Cloth(xyz0, tri, quad)
    mass = 1.0 / cl.np
    bc_h = DC.pin_two_corners(c["ndiv"])
    bc = torch.tensor(bc_h, device=dev)
    E = torch.full((cl.ntri,), c["young"], dtype=torch.float64, device=dev)
    X0 = torch.tensor(xyz0, device=dev)
    rng = np.random.default_rng(c["target_seed"])
    target = X0 + torch.tensor(rng.standard_normal(xyz0.size) * c["target_sigma"], device=dev)
    step_args = (c["nu"], c["stiff_bend"], c["g"], mass, c["dt"], c["tol"], c["max_iter"])
    x, v = X0.clone(), torch.zeros_like(X0)
    cl.StepTime_InternalDynamicsILU(x, v, bc, E, *step_args)  # warm-up
    x, v = X0.clone(), torch.zeros_like(X0)
    e0, e1, e2 = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    torch.cuda.synchronize()
    e0.record()
    st = cl.rollout(x, v, bc, E, *step_args, nsteps, c["ckpt_every"])
    e1.record()
    xbar, vbar = (x - target).contiguous(), torch.zeros_like(x)
    dLdE = torch.zeros(cl.ntri, dtype=torch.float64, device=dev)
    sb = cl.rollout_adjoint(xbar, vbar, dLdE)
    e2.record()
    torch.cuda.synchronize()
    fwd_ms, adj_ms = e0.elapsed_time(e1), e1.elapsed_time(e2)
    out = {"workload": f"implicit cloth, {cl.np} vertices, {cl.ntri} triangles, {cl.nquad} bending quads, "
                       f"backward Euler dt={c['dt']}, FP64 ILU(0)-PCG tol {c['tol']} capped at {c['max_iter']} "
                       f"iterations per step, checkpoints every {c['ckpt_every']} steps",
           "steps_timed": nsteps, "steps_in_workload": c["nsteps"],
           "ms_per_step": round(fwd_ms / nsteps, 3), "pcg_iterations_per_step": st.iterations / nsteps,
           "ms_per_step_and_pcg_iteration": round(fwd_ms / max(st.iterations, 1), 3),
           "max_rel_residual": st.rel_residual, "forward_ms": round(fwd_ms, 2), "adjoint_ms": round(adj_ms, 2),
           "adjoint_over_forward": round(adj_ms / fwd_ms, 3), "adjoint_pcg_iterations": sb.iterations,
           "gradient_finite": bool(torch.isfinite(dLdE).all())}
    if c["ndiv"] >= 64:
        out["note"] = ("ILU(0) of this system amplifies by >1e20 at >= 64x64 cells (the reference's own "
                       "factorisation: 1.5e20 at 64 cells, 2.4e122 at 255), so every step runs its 100-iteration cap "
                       "without converging; correctness and gradients are tested at <= 48x48 cells")
    if cpu:
        from oracle import port
        from oracle import cloth as OC
        O = port()
        ind, psup = O.psup(quad, 4, cl.np)
        t = time.perf_counter()
        _, _, nh = OC.cloth_step(O, ind, psup, xyz0, np.zeros_like(xyz0), xyz0, bc_h, tri, quad,
                                 np.full(cl.ntri, c["young"]), c["nu"], c["stiff_bend"], np.array(c["g"]), mass,
                                 c["dt"], c["tol"], c["max_iter"])
        cpu_ms = (time.perf_counter() - t) * 1e3
        out["cpu_baseline"] = {"value": round(cpu_ms, 1), "unit": "ms per step", "cores": 1, "kind": "port",
                               "sample": f"the first step (from rest) of the C restatement (assembly, ILU(0), "
                                         f"{nh - 1} PCG iterations) on the same sheet",
                               "ms_per_step_and_pcg_iteration": round(cpu_ms / max(nh - 1, 1), 3)}
    return out


def iluk_bench(dev):
    """ILU(k) (Initialize_ILUk) on the 64^3 voxel block (823,875 DOF, per-tet E log-uniform [0.1, 10], seed 2):
    symbolic pattern (host), CopyValue + Decompose, and Solve_PCG to 1e-10 in FP64 and mixed precision."""
    import torch
    import delfem2_gb300 as D
    a = D.voxel_problem_arrays(64, 64, 64, 1.0 / 64, seed=2, e_range=(0.1, 10.0))
    P = D.StaticElasticProblem(a)
    b = P.assemble(b=torch.zeros(a["np"] * 3, dtype=torch.float64, device=dev))
    out = {"workload": f"64x64x64 voxels x 6 tets, {a['np'] * 3} DOF, Solve_PCG to 1e-10 with ILU(k) factors",
           "matrix_blocks": int(a["psup"].size)}
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for k in (0, 1, 2):
        ilu = D.CPreconditionerILU()
        t = time.perf_counter()
        ilu.Initialize_ILUk(P.K, k)
        torch.cuda.synchronize()
        sym_s = time.perf_counter() - t
        e0.record()
        ilu.CopyValue(P.K)
        assert ilu.Decompose()
        e1.record()
        torch.cuda.synchronize()
        fac_ms = e0.elapsed_time(e1)
        r, x = b.clone(), torch.zeros_like(b)
        D.Solve_PCG(r.clone(), x, 1e-10, 20000, P.K, ilu)  # warm-up
        r, x = b.clone(), torch.zeros_like(b)
        e0.record()
        hist = D.Solve_PCG(r, x, 1e-10, 20000, P.K, ilu)
        e1.record()
        torch.cuda.synchronize()
        fp64_ms = e0.elapsed_time(e1)
        xm = torch.zeros_like(b)
        e0.record()
        st = D.Solve_PCG_Mixed(b, xm, 1e-10, P.K, ilu, method=METHOD)
        e1.record()
        torch.cuda.synchronize()
        out[f"k{k}"] = {"ilu_blocks": int(ilu.pattern()[0].size), "pattern_s": round(sym_s, 3),
                        "factor_ms": round(fac_ms, 2), "fp64_iterations": len(hist) - 1,
                        "fp64_ms": round(fp64_ms, 2), "mixed_iterations": st.iterations,
                        "mixed_ms": round(e0.elapsed_time(e1), 2), "mixed_rel_residual": st.rel_residual}
    return out


def bicgstab_bench(dev, cpu: bool):
    """Solve_PBiCGStab with ILU(0) on the 64^3 voxel block's elastic system to 1e-10, FP64 (the reference calls
    BiCGStab on this kind of 3x3-block elastic system, 603_Fem3DStiffwarp/main.cpp:218); the C restatement timed
    per iteration on the host."""
    import torch
    import delfem2_gb300 as D
    a = D.voxel_problem_arrays(64, 64, 64, 1.0 / 64, seed=2, e_range=(0.1, 10.0))
    P = D.StaticElasticProblem(a)
    b = P.assemble()
    assert P.factor()
    bd = torch.tensor(b, device=dev)
    r, x = bd.clone(), torch.zeros_like(bd)
    D.Solve_PBiCGStab(r, x, 1e-10, 5000, P.K, P.ilu)  # warm-up
    r, x = bd.clone(), torch.zeros_like(bd)
    st = D.SolveStats()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    hist = D.Solve_PBiCGStab(r, x, 1e-10, 5000, P.K, P.ilu, st)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1)
    out = {"workload": f"64x64x64 voxel block, {a['np'] * 3} DOF, ILU(0)-BiCGStab to 1e-10 (FP64)",
           "ms": round(ms, 2), "iterations": len(hist), "rel_residual": st.rel_residual}
    if cpu:
        from oracle import port
        O = port()
        vc, vd = P.K.get_values()
        col, dia = P.ilu.pattern()
        ivc, ivd = P.ilu.values()
        its = 3
        t = time.perf_counter()
        O.solve_pbicgstab(a["psup_ind"], a["psup"], vc, vd, a["psup_ind"], col, dia, ivc, ivd, b, 1e-300, its + 1)
        per = (time.perf_counter() - t) * 1e3 / its
        out["cpu_baseline"] = {"value": round(per * len(hist), 1), "unit": "ms", "cores": 1, "kind": "port",
                               "sample": f"{its} BiCGStab iterations of the C restatement ({per:.1f} ms each) "
                                         f"scaled to the GPU's {len(hist)} iterations"}
    return out


def poisson_bench(dev, arrays, cpu: bool):
    """Scalar Poisson (1x1 blocks) on the workload's tet mesh: MergeLinSys_Poission_MeshTet3D with alpha = 1,
    source = 1, the bottom face held at 0 and the top face at 1 (lifted into b), ILU(0)-PCG to 1e-10 in FP64 and
    with FP32 iterations / FP64 reliable updates; the C restatement's PCG timed per iteration on the host."""
    import torch
    import delfem2_gb300 as D
    a = arrays
    nb = int(a["np"])
    K = D.CMatrixSparse()
    K.Initialize(nb, 1, True)
    K.SetPattern(a["psup_ind"], a["psup"])
    mesh = D.TetMesh(K, a["xyz"], a["tet"])
    z = a["xyz"].reshape(-1, 3)[:, 2]
    top = z > z.max() - 1e-12
    bc = ((z < 1e-12) | top).astype(np.int32)
    bc_d = torch.tensor(bc, device=dev)
    val_d = torch.tensor(np.where(top, 1.0, 0.0), device=dev)
    b = torch.zeros(nb, dtype=torch.float64, device=dev)
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]

    def assemble_factor():
        b.zero_()
        K.setZero()
        mesh.assemble_poisson(1.0, 1.0, b, val_d)
        K.SetFixedBC(bc_d)
        D.setRHS_Zero(b, bc_d)
        ilu.CopyValue(K)
        assert ilu.Decompose()

    assemble_factor()  # warm-up
    ev[0].record()
    assemble_factor()
    ev[1].record()
    torch.cuda.synchronize()
    out = {"workload": f"scalar Poisson on the {nb}-node tet mesh of the headline ({nb} DOF, 1x1 blocks), "
                       "ILU(0)-PCG to 1e-10",
           "assemble_factor_ms": round(ev[0].elapsed_time(ev[1]), 2)}
    r, x = b.clone(), torch.zeros_like(b)
    D.Solve_PCG(r, x, 1e-10, 20000, K, ilu)  # warm-up
    r, x = b.clone(), torch.zeros_like(b)
    st = D.SolveStats()
    ev[2].record()
    hist = D.Solve_PCG(r, x, 1e-10, 20000, K, ilu, st)
    ev[3].record()
    torch.cuda.synchronize()
    out["fp64_ms"] = round(ev[2].elapsed_time(ev[3]), 2)
    out["fp64_iterations"] = len(hist) - 1
    out["fp64_rel_residual"] = st.rel_residual
    xm = torch.zeros_like(b)
    D.Solve_PCG_Mixed(b, xm, 1e-10, K, ilu, method=METHOD, refresh=WORKLOAD["refresh"], max_iter=20000)
    xm.zero_()
    ev[2].record()
    sm = D.Solve_PCG_Mixed(b, xm, 1e-10, K, ilu, method=METHOD, refresh=WORKLOAD["refresh"], max_iter=20000)
    ev[3].record()
    torch.cuda.synchronize()
    out["mixed_ms"] = round(ev[2].elapsed_time(ev[3]), 2)
    out["mixed_iterations"] = sm.iterations
    out["mixed_rel_residual"] = sm.rel_residual
    if cpu:
        from oracle import port
        O = port()
        vc, vd = K.get_values()
        col, dia = ilu.pattern()
        ivc, ivd = ilu.values()
        its = 5
        t = time.perf_counter()
        O.nd_solve_pcg(1, a["psup_ind"], a["psup"], vc, vd, a["psup_ind"], col, dia, ivc, ivd, b.cpu().numpy(),
                       1e-300, its)
        per = (time.perf_counter() - t) * 1e3 / its
        out["cpu_baseline"] = {"value": round(per * out["fp64_iterations"], 1), "unit": "ms", "cores": 1,
                               "kind": "port",
                               "sample": f"{its} PCG iterations of the C restatement ({per:.1f} ms each) scaled to "
                                         f"the GPU's {out['fp64_iterations']} FP64 iterations"}
    return out


def run_ours(args):
    import torch
    import delfem2_gb300 as D
    from delfem2_gb300 import _native as N

    world, rank, local, dist = dist_setup(args)
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    w = SMALL if args.small else WORKLOAD
    P, arrays, setup = build_problem(w)
    ndof = P.ndof
    nz = int(arrays["psup"].size)
    nb = int(arrays["np"])
    lib = N.load()

    t0 = time.perf_counter()
    b = P.assemble(b=torch.zeros(ndof, dtype=torch.float64, device=dev))
    torch.cuda.synchronize()
    t1 = time.perf_counter()
    assert P.factor()
    torch.cuda.synchronize()
    t2 = time.perf_counter()
    setup.update(assemble_s=t1 - t0, ilu_s=t2 - t1)

    def solve_mixed():
        x = torch.zeros_like(b)
        st = D.Solve_PCG_Mixed(b, x, w["tol"], P.K, P.ilu, inner_tol=w["inner_tol"], method=METHOD,
                              refresh=w["refresh"])
        return x, st

    for k in range(args.warmup):
        t = time.perf_counter()
        x, st = solve_mixed()
        torch.cuda.synchronize()
        if k == 0:  # the first solve also builds the sweep schedules (tile partitions, records) once
            setup.update(first_solve_s=time.perf_counter() - t)
        elif k == 1:
            setup.update(second_solve_s=time.perf_counter() - t)
    if dist is not None:
        dist.barrier()
    clocks = ClockSampler(local)
    clocks.start()
    c0 = D._native.C.c_ulonglong(0)
    lib.dfm2g_launch_count(D._native.C.byref(c0))
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    ev0.record()
    stats = []
    for _ in range(args.steps):
        x, st = solve_mixed()
        stats.append((st.iterations, st.outer, st.rel_residual, st.ms))
    ev1.record()
    torch.cuda.synchronize()
    c1 = D._native.C.c_ulonglong(0)
    lib.dfm2g_launch_count(D._native.C.byref(c1))
    clk = clocks.stop()
    if dist is not None:
        dist.barrier()
    ms = ev0.elapsed_time(ev1) / args.steps
    ms = reduce_max(dist, ms, dev)
    launches = int(c1.value - c0.value)

    # plain FP64 GPU Solve_PCG on the same system (same metric, FP64 path)
    xf = torch.zeros_like(b)
    r = b.clone()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    hist64 = D.Solve_PCG(r, xf, w["tol"], 20000, P.K, P.ilu)
    e1.record()
    torch.cuda.synchronize()
    fp64_ms = e0.elapsed_time(e1)
    it64 = len(hist64) - 1

    # classic restarted refinement (a fresh FP32 PCG to inner_tol per FP64 step), for comparison
    xr = torch.zeros_like(b)
    e0.record()
    st_alt = D.Solve_PCG_Mixed(b, xr, w["tol"], P.K, P.ilu, inner_tol=w["inner_tol"], method=OTHER,
                               max_iter=4 * it64, allow_not_converged=True)
    e1.record()
    torch.cuda.synchronize()
    alt_ms = e0.elapsed_time(e1)

    # accuracy: vs the FP64 GPU solution, and vs the reference's golden sample when present
    xn = x.double().cpu().numpy()
    err_fp64 = float(np.linalg.norm(xn - xf.cpu().numpy()) / np.linalg.norm(xf.cpu().numpy()))
    err_oracle = None
    gpath = os.path.join(ROOT, "tests", "golden", "cfg3.npz")
    if not args.small and os.path.exists(gpath):
        g = np.load(gpath)
        err_oracle = float(np.abs(xn[g["idx"]] - g["x_sample"]).max() / np.abs(g["x_sample"]).max())

    # adjoint / forward: forward = assemble + factor + solve; adjoint = solve
    # K lam = dL/du on the same factors + the dL/dE element kernel
    g_u = (x - 0.9 * x).contiguous()
    ef0, ef1, ea1 = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    ef0.record()
    P.assemble(b=b)
    P.factor()
    xx, _ = solve_mixed()
    ef1.record()
    lam = torch.zeros_like(b)
    D.Solve_PCG_Mixed(g_u, lam, w["tol"], P.K, P.ilu, inner_tol=w["inner_tol"], method=METHOD,
                              refresh=w["refresh"])
    dLdE = torch.zeros(arrays["ntet"], dtype=torch.float64, device=dev)
    P.mesh.dLdE(w["nu"], xx, lam, dLdE)
    ea1.record()
    torch.cuda.synchronize()
    fwd_ms, adj_ms = ef0.elapsed_time(ef1), ef1.elapsed_time(ea1)

    # e2e: the public C-ABI call with HOST buffers (H2D of b and D2H of x inside)
    bh = b.cpu().numpy().copy()
    xh = np.zeros_like(bh)
    D.Solve_PCG_Mixed(bh, xh, w["tol"], P.K, P.ilu, inner_tol=w["inner_tol"], method=METHOD,
                              refresh=w["refresh"])
    if dist is not None:
        dist.barrier()
    t = time.perf_counter()
    for _ in range(args.steps):
        D.Solve_PCG_Mixed(bh, xh, w["tol"], P.K, P.ilu, inner_tol=w["inner_tol"], method=METHOD,
                              refresh=w["refresh"])
    torch.cuda.synchronize()
    e2e_ms = reduce_max(dist, (time.perf_counter() - t) * 1e3 / args.steps, dev)

    # per-kernel device time (CUDA events around every launch, one extra solve)
    lib.dfm2g_profile_reset()
    lib.dfm2g_profile_enable(1)
    solve_mixed()
    lib.dfm2g_profile_enable(0)
    prof = {}
    for k, name in enumerate(N.PROF_KINDS):
        cnt, tot = D._native.C.c_uint(0), D._native.C.c_double(0)
        lib.dfm2g_profile_read(k, D._native.C.byref(cnt), D._native.C.byref(tot))
        if cnt.value:
            prof[name] = {"launches": cnt.value, "ms_total": tot.value, "ms_avg": tot.value / cnt.value}
    hbm, peak_kind = peaks()
    dom = max((k for k in prof if k in ("spmv", "fwd", "bwd", "update", "dot", "pupdate")),
              key=lambda k: prof[k]["ms_total"])
    alg = algorithmic_bytes(dom, nb, nz, 4)
    achieved = alg / (prof[dom]["ms_avg"] * 1e-3) / 1e9
    per_kernel = {k: dict(v, gbs=(algorithmic_bytes(k, nb, nz, 4) / (v["ms_avg"] * 1e-3) / 1e9
                                  if k != "outer" else None)) for k, v in prof.items()}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        it_sample = args.cpu_iters
        ms_it = cpu_port_ms_per_iter(P, b.cpu().numpy(), it_sample)
        cpu = {"value": ms_it * it64, "unit": "ms", "cores": 1, "kind": "port",
               "sample": f"{it_sample} Solve_PCG iterations of the C restatement on the same "
                         f"{ndof}-DOF system ({ms_it:.1f} ms/iteration), scaled to the {it64} "
                         f"iterations the FP64 solve takes to 1e-10",
               "host_cores_available": os.cpu_count()}
        if not args.small and not args.no_cpu_full_solve:
            cpu["full_solve_check"] = cpu_full_solve_cfg2(it_sample)

    its = [s[0] for s in stats]
    out = {
        "metric": METRIC, "value": round(ms, 3), "unit": "ms", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms, 3), "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
        "data": "synthetic: voxel tet mesh, seeded log-uniform per-tet E, body force, z=0 clamped",
        "config": {"workload": f"static linear elasticity, {w['nx']}x{w['ny']}x{w['nz']} voxels x 6 tets, "
                               f"{ndof} DOF, ILU(0)-PCG in FP32 with FP64 reliable updates (refresh factor "
                               f"{w['refresh']}) to |b - Ku|/|b| < {w['tol']}",
                   "dof": ndof, "nblk": nb, "nnz_blocks": nz, "tets": arrays["ntet"],
                   "l2": "inputs larger than L2 (FP32 K 0.57 GB, FP64 K 1.15 GB, factors 1.7 GB)",
                   "parallelism": f"replicas x{world}"},
        "iterations_inner": int(np.median(its)), "outer_steps": int(stats[-1][1]),
        "rel_residual": stats[-1][2], "err_vs_fp64_gpu": err_fp64, "err_vs_reference_sample": err_oracle,
        "fp64_ms": round(fp64_ms, 3), "fp64_iterations": it64,
        "speedup_vs_fp64": round(fp64_ms / ms, 3),
        "refinement": ("reliable updates: one FP32 PCG (FP32 K, FP32 ILU, FP64 alpha/beta); the FP32 iterate is "
                       "flushed into the FP64 solution and the residual recomputed in FP64 (FP64 K) each time "
                       f"|r| drops by the factor {w['refresh']}; the restarted scheme (a fresh FP32 PCG to "
                       f"inner_tol {w['inner_tol']} per FP64 step) is reported as restart_refinement_*"),
        "restart_refinement_ms": round(alt_ms, 3), "restart_refinement_iterations": st_alt.iterations,
        "restart_refinement_rel_residual": st_alt.rel_residual,
        "restart_refinement_speedup_vs_fp64": round(fp64_ms / alt_ms, 3),
        "dof_iter_per_s": ndof * float(np.median(its)) / (ms * 1e-3),
        "adjoint_over_forward": round(adj_ms / fwd_ms, 3), "forward_ms": round(fwd_ms, 3),
        "adjoint_ms": round(adj_ms, 3),
        "e2e": {"value": round(e2e_ms, 3), "unit": "ms", "h2d_bytes_per_step": 8 * ndof,
                "d2h_bytes_per_step": 8 * ndof},
        "roofline": {"bound": "hbm", "kernel": dom, "achieved": round(achieved, 1), "peak": hbm,
                     "peak_source": peak_kind, "unit": "GB/s", "frac": round(achieved / hbm, 4),
                     "algorithmic_bytes_per_launch": alg, "traffic": traffic_from_profiles(dom)},
        "kernels": per_kernel,
        "cpu_baseline": cpu, "clocks": clk, "gpu_launches": launches, "setup": setup,
    }
    if args.cloth_steps > 0:
        cpu_ok = rank == 0 and world == 1 and not args.no_cpu_baseline
        out["cloth"] = cloth_bench(dev, args.cloth_steps, cpu_ok)
        out["cloth_converging"] = cloth_bench(dev, CLOTH_CONVERGING["nsteps"], cpu_ok, CLOTH_CONVERGING)
    if not args.no_iluk:
        out["ilu_k"] = iluk_bench(dev)
        out["bicgstab"] = bicgstab_bench(dev, rank == 0 and world == 1 and not args.no_cpu_baseline)
        out["poisson"] = poisson_bench(dev, arrays, rank == 0 and world == 1 and not args.no_cpu_baseline)
    if rank == 0:
        print(json.dumps(out))
    if dist is not None:
        dist.destroy_process_group()


def run_reference(args):
    """The reference's CPU Solve_PCG (oracle/_ref where it was built here, else
    the C restatement), timed on this host; each step is a bounded sample of
    PCG iterations on the same system, scaled to the full solve."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import oracle
    w = SMALL if args.small else WORKLOAD
    try:
        O = oracle.reference()
        kind = "reference"
    except Exception:
        O = oracle.port()
        kind = "port"
    t0 = time.perf_counter()
    xyz, tet = O.voxel_tet_mesh(w["nx"], w["ny"], w["nz"], w["h"])
    np_ = xyz.size // 3
    ind, psup = O.psup(tet, 4, np_)
    rng = np.random.default_rng(w["seed"])
    young = np.exp(rng.uniform(np.log(w["e_lo"]), np.log(w["e_hi"]), tet.size // 4))
    vc, vd, b = np.zeros(psup.size * 9), np.zeros(np_ * 9), np.zeros(np_ * 3)
    O.assemble_tet_linear(ind, psup, vc, vd, b, xyz, tet, young, w["nu"], w["rho"], list(w["g"]))
    bc = np.zeros(np_ * 3, np.int32)
    bc[np.repeat(xyz[2::3] == 0.0, 3)] = 1
    O.set_fixed_bc(ind, psup, vc, vd, bc)
    O.rhs_zero(b, bc)
    col, dia = O.ilu_pattern0(ind, psup)
    ivc, ivd = O.ilu_copy_value(ind, col, psup, vc, vd)
    O.ilu_decompose(ind, col, dia, ivc, ivd)
    setup_s = time.perf_counter() - t0
    gpath = os.path.join(ROOT, "tests", "golden", "cfg3.npz")
    n_full = None
    if not args.small and os.path.exists(gpath):
        n_full = iterations_to(np.load(gpath)["hist"], w["tol"])
    if n_full is None:  # run the full solve once to know the count (small workload)
        _, _, h = O.solve_pcg(ind, psup, vc, vd, col, dia, ivc, ivd, b, w["tol"], 100000)
        n_full = len(h) - 1
    per = args.cpu_iters
    for _ in range(args.warmup):
        O.solve_pcg(ind, psup, vc, vd, col, dia, ivc, ivd, b, 1e-300, 1)
    t = time.perf_counter()
    for _ in range(args.steps):
        O.solve_pcg(ind, psup, vc, vd, col, dia, ivc, ivd, b, 1e-300, per)
    ms_it = (time.perf_counter() - t) * 1e3 / (args.steps * per)
    value = ms_it * n_full
    sample = (f"{per} Solve_PCG iterations per step ({ms_it:.1f} ms/iteration, 1 core, serial by construction) "
              f"scaled to the {n_full} iterations FP64 ILU(0)-PCG needs to {w['tol']}")
    out = {"impl": "reference", "metric": METRIC, "value": round(value, 1), "unit": "ms", "n_gpus": world,
           "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(value, 1), "higher_is_better": False,
           "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (same as ours)",
           "config": {"workload": f"{w['nx']}x{w['ny']}x{w['nz']} voxels x 6 tets, {np_ * 3} DOF, FP64 "
                                  f"ILU(0)-PCG to {w['tol']}", "dof": np_ * 3},
           "cpu_baseline": {"value": round(value, 1), "unit": "ms", "cores": 1, "kind": kind, "sample": sample,
                            "host_cores_available": os.cpu_count(), "setup_s": round(setup_s, 2)},
           "e2e": {"value": round(value, 1), "unit": "ms", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--small", action="store_true", help="32x32x16 voxels instead of 128x128x64")
    ap.add_argument("--cpu-iters", type=int, default=6)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-cpu-full-solve", action="store_true",
                    help="skip the fully timed 64^3 CPU solve that checks the CPU projection")
    ap.add_argument("--no-iluk", action="store_true", help="skip the ILU(k) line")
    ap.add_argument("--cloth-steps", type=int, default=20,
                    help="steps of the 100-step cloth workload to time (0: skip the cloth line)")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
