#!/usr/bin/env python
"""Benchmark of the 3D spherical iBEM hot path on GB300.

Workload (one "step" = one time-to-solution of one microstructure): 2,000 spheres,
radius U[0.8, 1.2] x 0.012, random sequential addition with a surface gap >= 0.1 r,
volume fraction ~15%, matrix E = 70 GPa / nu = 0.3, particles E = 400 GPa / nu = 0.2,
linear Taylor eigenstrain (24 unknowns per sphere, N = 48,000), remote uniaxial stress
sigma33 = 1, stresses on a cell-centred 64^3 grid (262,144 points).  Seeded synthetic
inputs (no dataset is involved).

A step = far-field right-hand side + solve + stresses at all grid points (double-float
sphere sums, ~48 bits).  The chosen form (default, --form learned_gmres) solves without
storing the matrix: FP32 restarted GMRES on the scaled system with on-the-fly pair-block
products, right-preconditioned by block-Jacobi plus GNN-weighted Neumann blocks on the
16-nearest-neighbour graph, inside FP64 iterative refinement whose residuals are FP64
on-the-fly products (stop: relative residual <= 1e-10).  The network is trained before
the timed region on small microstructures of the same distribution (its time is
reported).  --form mixed_ir times the dense path instead: FP64 pair assembly, FP32 LU with
split-BF16 tensor-core updates and FP64 GMRES-IR.  Both dense forms (mixed and plain FP64)
are also run once on the same microstructure and the chosen form's difference to the
plain FP64 solution is reported.  `value` is seconds per solution with inputs resident in
HBM; `e2e` is the same through the host-buffer C ABI (ibem_e3d_run_host_mf, or
ibem_e3d_run_host for mixed_ir) with inputs copied in and X / stresses copied out inside
the timed region.

--impl reference times the CPU restatement of the reference's algorithm (the oracle,
OpenMP over all host cores) on bounded samples of the same workload, extrapolated to it.
"""
from __future__ import annotations

import argparse
import ctypes
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

METRIC = "time-to-solution at 1e-8 rel. error: chosen form vs plain FP64, 1xGB300"
WORKLOAD = "2000 spheres r~U[0.8,1.2]*0.012, vf 15%, linear eigenstrain (N=48000), far-field sigma33=1, 64^3 grid"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--num", type=int, default=2000)
    ap.add_argument("--grid", type=int, default=64)
    ap.add_argument("--tol", type=float, default=1e-12)
    ap.add_argument("--no-plain", action="store_true", help="skip the one plain-FP64 comparison solve")
    ap.add_argument("--e2e-steps", type=int, default=5)
    ap.add_argument("--form", default="learned_gmres", choices=["learned_gmres", "mixed_ir"])
    ap.add_argument("--train-steps", type=int, default=300)
    ap.add_argument("--batch", type=int, default=256, help="realisations of the batched measurement (0: skip)")
    ap.add_argument("--no-cube64", action="store_true", help="skip the bounded-cube (64 spheres) measurement")
    ap.add_argument("--no-cube64-cpu", action="store_true", help="skip the oracle timing of the bounded cube")
    ap.add_argument("--ellipsoids", type=int, default=4000, help="ellipsoids of the mixed-form measurement (0: skip)")
    ap.add_argument("--large", type=int, default=20000,
                    help="spheres of the vf-25%% learned vs block-Jacobi measurement at config 4's size (0: skip)")
    ap.add_argument("--ell-plain", type=int, default=1000,
                    help="ellipsoids of the plain-FP64 vs mixed comparison (0: skip)")
    ap.add_argument("--quad-form", default="mf", choices=["mf", "bj", "mixed"],
                    help="solver of the batch's quadratic realisations: matrix-free block-Jacobi GMRES (layout 60, "
                         "no matrices), or dense: block-Jacobi GMRES or FP32 LU + GMRES-IR")
    return ap.parse_args()


def make_case(num, grid, seed):
    from ibemproject_gb300 import cases
    return cases.farfield_case(num=num, r0=0.012, vf=0.15, grid=grid, seed=seed)


# ------------------------------------------------------------------ CPU baseline (oracle)
def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    oracle.build()
    return oracle


def lu_calibration(case, sizes=(2400, 4800)):
    """Full-pivot LU (the reference's fullPivLu algorithm, oracle restatement) of the leading
    sub-systems of N = sizes[k] unknowns: seconds per size and the fitted exponent."""
    oracle = _oracle()
    m = oracle.mat(case.E0, case.nu0, case.E1, case.nu1)
    ts = []
    for n in sizes:
        ns = n // 24
        A = oracle.pair_blocks(case.centers[:ns], case.radius[:ns], m, 24)
        b = oracle.farfield_rhs(ns, m, 24, case.sig_inf)
        t = time.perf_counter()
        oracle.solve_fullpiv(A, b)
        ts.append(time.perf_counter() - t)
    expo = float(np.log(ts[-1] / ts[0]) / np.log(sizes[-1] / sizes[0])) if len(sizes) > 1 else 3.0
    return {"N": list(sizes), "seconds": ts, "fitted_exponent": expo}


def cpu_baseline(case, lu=None, pair_spheres=200, points=256):
    """The oracle (CPU restatement, OpenMP over all host cores) on a fixed sample plan of the
    workload, extrapolated by the algorithm's own scaling: pair blocks of the first
    `pair_spheres` spheres (x (num / n)^2), the full-pivot LU at N = 4,800 (x (N / 4,800)^3;
    `lu` from lu_calibration, timed once) and the stress sums of `points` grid points over
    all spheres (x nump / points).  The same plan serves the bench's cpu_baseline leg and
    --impl reference, so the two report the same quantity."""
    oracle = _oracle()
    m = oracle.mat(case.E0, case.nu0, case.E1, case.nu1)
    num, N, nump = case.num, 24 * case.num, case.nump
    lu = lu or lu_calibration(case)
    ns = min(num, pair_spheres)
    t = time.perf_counter()
    oracle.pair_blocks(case.centers[:ns], case.radius[:ns], m, 24)
    ta = time.perf_counter() - t
    t_asm = ta * (num / ns) ** 2
    t_sol = lu["seconds"][-1] * (N / lu["N"][-1]) ** 3
    E = np.zeros(N)
    E[0::24] = 1e-12
    npts = min(points, nump)
    idx = np.linspace(0, nump - 1, npts).astype(int)
    t = time.perf_counter()
    oracle.post(case, 24, E, sig_inf=case.sig_inf, points=case.points[idx])
    tf = time.perf_counter() - t
    t_fld = tf * nump / npts
    total = t_asm + t_sol + t_fld
    cores = int(os.environ.get("OMP_NUM_THREADS", os.cpu_count() or 1))
    return {
        "value": total, "unit": "s", "cores": cores, "kind": "port",
        "sample": (f"oracle (CPU restatement of the reference, OpenMP) timed on the pair blocks of {ns} of {num} "
                   f"spheres (x (num/{ns})^2), full-pivot LU at N={lu['N'][-1]} (x (N/{lu['N'][-1]})^3; fitted exponent "
                   f"{lu['fitted_exponent']:.2f} between N={lu['N'][0]} and {lu['N'][-1]}), stress sums at {npts} of "
                   f"{nump} grid points over all spheres (x {nump}/{npts}); extrapolated"),
        "extrapolated": True,
        "stages_s": {"assembly": t_asm, "solve": t_sol, "field": t_fld},
        "measured_s": {"pair_blocks": ta, "lu": lu["seconds"], "field": tf},
        "lu_calibration": lu,
    }


def cube64_cpu(case, points=64):
    """The oracle on the bounded-cube workload at 24 unknowns per sphere: assembly (every
    block, ApplyBC) and the full-pivot LU measured in full; the stresses measured at `points`
    of the 32^3 grid points and scaled to all of them (the cost is the same per point)."""
    oracle = _oracle()
    m = oracle.mat(case.E0, case.nu0, case.E1, case.nu1)
    t = time.perf_counter()
    H, G = oracle.assemble(case, 24, m)
    A, b, tcol, _ = oracle.apply_bc(case, H, G)
    t_asm = time.perf_counter() - t
    t = time.perf_counter()
    X = oracle.solve_fullpiv(A, b)
    t_sol = time.perf_counter() - t
    U, T = oracle.get_ut(case, tcol, X)
    idx = np.linspace(0, case.nump - 1, points).astype(int)
    t = time.perf_counter()
    oracle.post(case, 24, X[3 * case.NN:], U, T, points=case.points[idx], m=m)
    t_post = (time.perf_counter() - t) * case.nump / points
    cores = int(os.environ.get("OMP_NUM_THREADS", os.cpu_count() or 1))
    return {"value": t_asm + t_sol + t_post, "unit": "s", "cores": cores, "kind": "port",
            "sample": (f"oracle at 24 unknowns per sphere: assembly + ApplyBC and full-pivot LU (N={len(b)}) measured "
                       f"in full; stresses at {points} of {case.nump} grid points, scaled by {case.nump}/{points}"),
            "stages_s": {"assembly": t_asm, "solve": t_sol, "field": t_post}}


# ------------------------------------------------------------------ roofline
def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return d.get("hbm_gbs", 6800.0), d.get("bf16_tflops_sustained", 1700.0), "measured"
    return 6800.0, 1700.0, "fallback"


# DRAM bytes (read + write) per launch of k_umma_bf16x3 over every launch of this workload,
# from one ncu capture of the bench command (profiles/k_umma_bf16x3_bench2000_traffic.md)
UMMA_TRAFFIC_BYTES_PER_LAUNCH = 242.7e6


def roofline(prof):
    """Roofline of the tensor-core GEMM (the trailing updates of the factorisation, the
    largest kernel of the step): achieved = algorithmic flops (2 m n k per launch, the FP32
    GEMM's work) / its event-timed duration, against the measured sustained dense BF16 rate.
    The split-BF16 scheme issues 3 BF16 MMAs per product, so frac_of_issued (3x) is the
    fraction of the tensor pipe's rate actually used."""
    hbm, tf, src = measured_peaks()
    g = prof.get("gemm_tc")
    if not g or g["ms"] <= 0:
        return None
    achieved = g["flops"] / (g["ms"] * 1e-3) / 1e12
    return {"kernel": "k_umma_bf16x3 (gemm_tc)", "bound": "tensor", "achieved": achieved, "peak": tf,
            "unit": "TFLOP/s", "frac": achieved / tf, "peak_source": f"{src} bf16_tflops_sustained",
            "launches": g["launches"], "avg_launch_ms": g["ms"] / max(1, g["launches"]),
            "flops_per_launch": g["flops"] / max(1, g["launches"]),
            "tensor_flops_issued_per_launch": 3 * g["flops"] / max(1, g["launches"]),
            "frac_of_issued": 3 * achieved / tf,
            "traffic": UMMA_TRAFFIC_BYTES_PER_LAUNCH, "traffic_unit": "bytes per launch (ncu dram read+write)",
            "traffic_source": "profiles/k_umma_bf16x3_bench2000_traffic.md"}


def sm_count():
    import torch
    return int(torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count)


def roofline_chosen(prof, case):
    """Roofline of the largest stage of the matrix-free step, the split stress sums
    (field24_far, FP32 beyond 12 radii of a warp's points, and field24_near, double-float
    within): FP32-pipe bound.  Algorithmic work = FIELD_ALG_FLOPS_PER_PAIR, the FP32 flops of
    the contracted strain of one (point, sphere) pair, x the pairs of one call, over the
    event-timed duration of the call (the two kernels plus the Morton sort of the points);
    the executed-flop fraction (ncu's FP32 instruction count of both kernels, double-float
    arithmetic near the points included) is reported beside it.  Peak = the nominal FP32 FMA
    rate (SMs of this device x 128 lanes x 2 flops) at the measured maximum SM clock;
    MEASURED_PEAKS.json holds no FP32 figure."""
    f = prof.get("field")
    if not f or f["ms"] <= 0:
        return None
    mhz = 2070.0
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as fh:
            mhz = json.load(fh).get("sm_max_mhz", mhz)
    nsm = sm_count()
    peak = nsm * 128 * 2 * mhz * 1e6 / 1e12
    pairs = case.nump * case.num
    launch_s = f["ms"] / f["launches"] * 1e-3
    achieved = FIELD_ALG_FLOPS_PER_PAIR * pairs / launch_s / 1e12
    executed = FIELD_DF_FLOPS_PER_PAIR * pairs / launch_s / 1e12
    return {"kernel": "field24_far + field24_near (stress sums, FP32 far / double-float near)", "bound": "fp32",
            "achieved": achieved, "peak": peak, "unit": "TFLOP/s", "frac": achieved / peak,
            "peak_source": f"nominal FP32 FMA rate, {nsm} SMs at sm_max_mhz {mhz:g} (no measured FP32 peak)",
            "sm_count": nsm, "flops_per_pair": FIELD_ALG_FLOPS_PER_PAIR,
            "flops_per_pair_note": "algorithmic: the FP32 contraction of one (point, sphere) pair",
            "executed_flops_per_pair": FIELD_DF_FLOPS_PER_PAIR, "executed_achieved": executed,
            "frac_executed": executed / peak, "pairs_per_launch": pairs,
            "avg_launch_ms": f["ms"] / f["launches"], "traffic": FIELD_DF_TRAFFIC_PER_LAUNCH,
            "traffic_unit": "bytes per call (ncu dram read+write of both kernels)",
            "traffic_source": FIELD_DF_SOURCE, "flops_source": FIELD_DF_SOURCE}


# Algorithmic FP32 flops of one (point, sphere) pair of the contracted stress sum: the FP32
# path alone (FADD + FMUL + 2 FFMA thread instructions counted by ncu on a field24_far launch
# whose points are far from every sphere, 2.431e10 flops / 6.554e7 pairs).
FIELD_ALG_FLOPS_PER_PAIR = 370.9
# Executed FP32 flops per pair on this workload (the same count over both kernels of one
# full-size call, double-float within 12 radii: 1.731e11 far + 1.419e11 near = 3.150e11 /
# 5.243e8 pairs) and the call's DRAM bytes (read + write of both kernels) from the same capture.
FIELD_DF_FLOPS_PER_PAIR = 600.8
FIELD_DF_TRAFFIC_PER_LAUNCH = 43.97e6
FIELD_DF_SOURCE = "profiles/kernels_small_cases.md"


# ------------------------------------------------------------------ clocks
class Clocks:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                                          "-i", str(self.index), "-lms", "200"], stdout=open(self.path, "w"),
                                         stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        rows = []
        for ln in open(self.path):
            p = [x.strip() for x in ln.split(",")]
            if len(p) >= 9:
                rows.append(p)
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


# ------------------------------------------------------------------ replicas
def job_seconds_per_solution(ms_local, world, device=None):
    """Whole-job seconds per solution of N replicas: every rank solved one realisation in
    its own timed steps; the job's time is the slowest rank's, and N solutions came out of
    it (weak scaling).  Single process: ms_local / 1e3."""
    if world <= 1:
        return ms_local / 1e3
    import torch
    t = torch.tensor([float(ms_local)], dtype=torch.float64, device=device)
    torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    return float(t.item()) / 1e3 / world


# ------------------------------------------------------------------ ours
def train_preconditioner(args, rank, dev):
    """GNN weights of the learned preconditioner, trained on 12 microstructures of 100-150
    spheres (radius U[0.8, 1.2] x 0.012, volume fraction U[10%, 20%], contrast E1/E0
    U[2, 20], four of them at the bench's own 400/70), residual / correction pairs from the
    plain FP64 solver, 4 per microstructure.  Returns (params tensor, info dict)."""
    from ibemproject_gb300 import batch as B
    from ibemproject_gb300 import cases
    t = time.perf_counter()
    rng = np.random.default_rng(77 + rank)
    nums = rng.integers(100, 151, size=12)
    vfs = rng.uniform(0.10, 0.20, size=12)
    contrast = rng.uniform(2.0, 20.0, size=12)
    contrast[:4] = 400.0 / 70.0   # the bench microstructure's own contrast
    train = [cases.farfield_case(num=int(n), r0=0.012, vf=float(v), grid=0, seed=9000 + 31 * rank + k,
                                 E1=70e9 * float(c))
             for k, (n, v, c) in enumerate(zip(nums, vfs, contrast))]
    bt = B.DeviceBatch(train, device=dev)
    r, e = B.training_pairs(bt, nrhs=4, seed=5 + rank)
    t_data = time.perf_counter() - t
    params = B.init_params(seed=1, device=dev)
    t = time.perf_counter()
    hist = B.train(bt, r, e, params, steps=args.train_steps, lr=3e-3)
    t_train = time.perf_counter() - t
    info = {"microstructures": len(train), "spheres": int(sum(nums)), "pairs": 4 * len(train),
            "steps": args.train_steps, "loss_first": float(hist[0]), "loss_last": float(hist[-1]),
            "data_s": t_data, "train_s": t_train, "params": int(params.numel())}
    return params, info


def run_batched(args, dev, params):
    """Batched realisations (config 5): args.batch microstructures of U[50, 500] particles,
    spheres or ellipsoids 50/50 (spheres: radius U[0.8, 1.2] x 0.008, min gap 0.1 r;
    ellipsoids: a1 = 0.008, a2 = a1 U[0.5, 1], a3 = a1 U[0.25, 1], Haar orientations, gap
    ~0.2 a3; both packed by the library's hard-particle Monte Carlo generators), volume
    fraction U[10%, 30%], contrast E1/E0 U[2, 20]; spheres half with linear eigenstrain (24
    unknowns per sphere) and half with quadratic (60), ellipsoids linear; uniaxial remote
    stress.  One step = right-hand sides, the linear sphere realisations in one batched
    matrix-free solve (learned preconditioner, FP64 refinement to relative residual 1e-10),
    the quadratic sphere realisations in one batched matrix-free solve of layout 60
    (block-Jacobi, the same refinement; --quad-form bj / mixed: assembled and solved densely
    like the ellipsoids), the ellipsoid realisations assembled (FP64 pair blocks) and solved
    one after another to scaled backward error 1e-12 (FP64 refinement of FP32-product GMRES
    with per-particle block-Jacobi), and the effective moduli of all.  Reports realisations per
    second."""
    import torch
    import ibemproject_gb300 as g
    from ibemproject_gb300 import batch as B
    from ibemproject_gb300 import cases
    rng = np.random.default_rng(4242)
    nums = rng.integers(50, 501, size=args.batch)
    vfs = rng.uniform(0.10, 0.30, size=args.batch)
    contrast = rng.uniform(2.0, 20.0, size=args.batch)
    ell = rng.random(args.batch) < 0.5
    quad = (rng.random(args.batch) < 0.5) & ~ell
    t = time.perf_counter()
    cs = [cases.ellipsoid_case(int(n), a1=0.008, vf=float(v), seed=7000 + k, E1=70e9 * float(c), method="mc")
          if e else cases.generated_case(int(n), 0.008, float(v), seed=7000 + k, E1=70e9 * float(c))
          for k, (n, v, c, e) in enumerate(zip(nums, vfs, contrast, ell))]
    t_gen = time.perf_counter() - t
    vol = np.array([float(c.title.split("=")[1]) ** 3 for c in cs])   # cube of side L
    li, qi, ei = np.flatnonzero(~quad & ~ell), np.flatnonzero(quad), np.flatnonzero(ell)
    bl = B.DeviceBatch([cs[i] for i in li], device=dev) if li.size else None
    bq = B.DeviceBatch([cs[i] for i in qi], device=dev, layout=60) if qi.size else None
    be = B.DeviceBatch([cs[i] for i in ei], device=dev) if ei.size else None
    sig = np.array([0, 0, 0, 0, 0, 1.0])
    stream = torch.cuda.current_stream(dev)
    qform = g.SOLVE_MIXED_IR if args.quad_form == "mixed" else g.SOLVE_GMRES_BJ

    def step():
        out = {}
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
        ev[0].record(stream)
        if bl is not None:
            b = B.farfield_rhs(bl, sig)
            x, reps = B.solve(bl, b, B.PRECOND_LEARNED, params=params)
            e, _ = B.effective_modulus(bl, x, sig, volume=vol[li])
            out["lin"] = (x, reps, e, b)
        ev[1].record(stream)
        for key, bt, idx in (("quad", bq, qi), ("ell", be, ei)):
            if bt is not None:
                b = B.farfield_rhs(bt, sig)
                if key == "quad" and args.quad_form == "mf":
                    x, reps = B.solve(bt, b, B.PRECOND_BLOCK_JACOBI)
                else:
                    x, reps = B.dense_batch_solve(bt, b, g.SOLVE_GMRES_BJ if key == "ell" else qform, tol=1e-12)
                e, _ = B.effective_modulus(bt, x, sig, volume=vol[idx])
                out[key] = (x, reps, e, b)
            ev[2 if key == "quad" else 3].record(stream)
        return out, ev

    step()   # warm-up
    torch.cuda.synchronize()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    k = max(1, min(3, args.steps))
    evs = []
    t0.record(stream)
    for _ in range(k):
        out, ev = step()
        evs.append(ev)
    t1.record(stream)
    torch.cuda.synchronize()
    ms = t0.elapsed_time(t1) / k
    ms_lin = statistics.median(e[0].elapsed_time(e[1]) for e in evs)
    ms_quad = statistics.median(e[1].elapsed_time(e[2]) for e in evs)
    ms_ell = statistics.median(e[2].elapsed_time(e[3]) for e in evs)
    # realisations of each kind against the plain FP64 LU of their own layout
    errs = {"linear_spheres": [], "quadratic_spheres": [], "linear_ellipsoids": []}
    for kind, key, bt, idx, lay in (("linear_spheres", "lin", bl, li, 24), ("quadratic_spheres", "quad", bq, qi, 60),
                                    ("linear_ellipsoids", "ell", be, ei, 24)):
        if bt is None:
            continue
        x, _, _, b = out[key]
        sub = nums[idx]
        picks = {int(np.argmin(sub)), int(np.argmin(np.abs(sub - 200))), int(np.argmax(sub))}
        for s_ in sorted(picks):
            rows = bt.seg_rows(s_)
            if key == "ell":
                c = cs[idx[s_]]
                c0 = cases.Case(c.E0, c.nu0, c.E1, c.nu1, c.nodes, c.conn, c.bc, c.tbc, c.centers, c.radius,
                                np.zeros((0, 3)), c.sig_inf, c.title, c.axes, c.quats)
                xd = torch.from_numpy(g.run_host_ell(c0, form=g.SOLVE_FP64)[0])
                errs[kind].append(float((x[rows].cpu() - xd).abs().max() / xd.abs().max()))
            else:
                xd = B.dense_solve(cs[idx[s_]], b[rows], device=dev, layout=lay)
                errs[kind].append(float((x[rows] - xd).abs().max() / xd.abs().max()))
    E0 = np.array([c.E0 for c in cs])
    e_all = np.zeros(args.batch)
    for key, idx in (("lin", li), ("quad", qi), ("ell", ei)):
        if key in out:
            e_all[idx] = out[key][2]
    ratio = e_all / E0
    quad_mf = args.quad_form == "mf"
    lin_reps = out["lin"][1] if bl is not None else []
    quad_reps = out["quad"][1] if bq is not None else []
    dense_reps = ([] if quad_mf else quad_reps) + (out["ell"][1] if be is not None else [])
    return {"workload": (f"{args.batch} realisations, U[50,500] particles, spheres (r~U[0.8,1.2]*0.008) or ellipsoids "
                         "(a1=0.008, a2=a1 U[0.5,1], a3=a1 U[0.25,1]) 50/50, vf U[10%,30%], E1/E0 U[2,20]; spheres half "
                         "linear (24/sphere, matrix-free learned GMRES) and half quadratic (60/sphere, " +
                         ("matrix-free block-Jacobi GMRES" if quad_mf else
                          "assembled, block-Jacobi FP32-product GMRES + FP64 refinement" if args.quad_form == "bj" else
                          "assembled, FP32 LU + BF16x3 + FP64 GMRES-IR") +
                         "), ellipsoids linear (assembled, block-Jacobi FP32-product GMRES + FP64 refinement), "
                         "far-field sigma33"),
            "value": args.batch / (ms / 1e3), "unit": "realisations/s", "ms_per_batch": ms,
            "ms_linear_spheres": ms_lin, "ms_quadratic_spheres": ms_quad, "ms_ellipsoids": ms_ell,
            "realisations_linear_spheres": int(li.size), "realisations_quadratic_spheres": int(qi.size),
            "realisations_ellipsoids": int(ei.size),
            "particles": int(nums.sum()), "unknowns": int(24 * nums[li].sum() + 60 * nums[qi].sum() + 24 * nums[ei].sum()),
            "arnoldi_steps_max": max((r.inner for r in lin_reps), default=0),
            "refinement_steps_max": max((r.outer for r in lin_reps), default=0),
            "rel_residual_max": max((r.rel_residual for r in lin_reps), default=0.0),
            "quadratic_matrix_free": quad_mf,
            "quadratic_arnoldi_steps_max": max((r.inner for r in quad_reps), default=0) if quad_mf else None,
            "quadratic_rel_residual_max": max((r.rel_residual for r in quad_reps), default=0.0) if quad_mf else None,
            "dense_backward_error_max": max((r.backward_error for r in dense_reps), default=0.0),
            "dense_gmres_iterations_max": max((r.iterations for r in dense_reps), default=0),
            "rel_err_vs_plain_fp64": errs,
            "effective_modulus_over_E0": {"mean": float(ratio.mean()), "min": float(ratio.min()),
                                          "max": float(ratio.max())},
            "generation_s": t_gen}


def run_large(args, dev, params):
    """The learned preconditioner at BASELINE config 4's size, with spheres (the matrix-free
    products take spheres): args.large spheres of radius U[0.8, 1.2] x 0.008 packed by the
    library's hard-sphere Monte Carlo generator to vf 25% (N = 24 x args.large), uniaxial
    remote stress; matrix-free FP32 GMRES(50) with FP64 refinement to relative residual 1e-10,
    preconditioned by the network trained for the headline (never trained on this size), by
    the same blocks with every weight 1 (analytic Neumann) and by block-Jacobi.  One warm-up
    and one timed solve each (CUDA events, inputs in HBM)."""
    import torch
    from ibemproject_gb300 import batch as B
    from ibemproject_gb300 import cases
    t = time.perf_counter()
    c = cases.generated_case(args.large, 0.008, 0.25, seed=515, method="mc")
    t_gen = time.perf_counter() - t
    bt = B.DeviceBatch([c], device=dev)
    b = B.farfield_rhs(bt, np.array([0, 0, 0, 0, 0, 1.0]))
    out = {"workload": f"{args.large} spheres r~U[0.8,1.2]*0.008, hard-sphere Monte Carlo to vf 25%, linear eigenstrain "
                       f"(N={24 * args.large}), far-field sigma33; matrix-free GMRES(50) + FP64 refinement to 1e-10",
           "generation_s": t_gen}
    xs = {}
    for key, pc, pp in (("learned", B.PRECOND_LEARNED, params), ("neumann", B.PRECOND_NEUMANN, None),
                        ("block_jacobi", B.PRECOND_BLOCK_JACOBI, None)):
        B.solve(bt, b, pc, params=pp)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        x, reps = B.solve(bt, b, pc, params=pp)
        e1.record()
        torch.cuda.synchronize()
        xs[key] = x
        out[key] = {"s": e0.elapsed_time(e1) / 1e3, "arnoldi_steps": reps[0].inner, "refinement_steps": reps[0].outer,
                    "rel_residual": reps[0].rel_residual}
    ref = xs["block_jacobi"]
    out["rel_diff_learned_vs_block_jacobi"] = float((xs["learned"] - ref).abs().max() / ref.abs().max())
    return out


def run_cube64(args, dev):
    """The bounded-cube workload (unit cube, 6 x 10 x 10 Q4 elements, 64 spheres of radius
    0.05 by random sequential addition, seed 12345, stresses on the 32^3 cell-centred grid)
    through the host-buffer C ABI (ibem_e3d_run_host: assembly, ApplyBC, solve, stresses,
    copies included), at the reference's 78 unknowns per sphere and at 24, in the plain FP64
    and the mixed form; errors against the reference's own solution and stresses (the
    committed fixture, 1,024 grid points) and the oracle's 24-unknown solution."""
    import ibemproject_gb300 as g
    from ibemproject_gb300 import cases
    z = np.load(os.path.join(ROOT, "tests", "golden", "cube64_reference.npz"))
    c = cases.bounded_cube_case(n_face=10, num=64, radius=0.05, grid=32, seed=12345)
    idx = z["subset"]
    n3 = 3 * c.NN
    runs = {}
    for name, layout, form in (("fp64_78", 78, g.SOLVE_FP64), ("mixed_78", 78, g.SOLVE_MIXED_IR),
                               ("fp64_24", 24, g.SOLVE_FP64), ("mixed_24", 24, g.SOLVE_MIXED_IR)):
        g.run_host(c, layout=layout, form=form, tol=1e-14)   # warm-up
        t = time.perf_counter()
        X, S, rep = g.run_host(c, layout=layout, form=form, tol=1e-14)
        dt = time.perf_counter() - t
        Xr, Sr = (z["X78"], z["stress78"]) if layout == 78 else (z["X24"], z["stress24"])
        E, Er = X[n3:].reshape(-1, layout), Xr[n3:].reshape(-1, layout)
        err_e = max(float(np.abs(E[:, a:b] - Er[:, a:b]).max() / np.abs(Er[:, a:b]).max())
                    for a, b in ((0, 6), (6, 24), (24, layout)) if b > a)
        runs[name] = {"time_to_solution_s": dt, "N": len(X), "backward_error": rep.backward_error,
                      "rel_err_eigenstrain_vs": "reference" if layout == 78 else "oracle",
                      "rel_err_eigenstrain": err_e,
                      "rel_err_stress": float(np.abs(S[idx] - Sr).max() / np.abs(Sr).max())}
    ref = {}
    for ln in str(z["ref_timings"]).splitlines():
        k, v = ln.split()
        ref[k] = float(v)
    asm = sum(v for k, v in ref.items() if k.startswith("add"))
    ref_total = ref.get("preprocess", 0) + asm + ref["ApplyBC"] + ref["solve"] + ref["getFlux"] * c.nump / len(idx)
    out = {"workload": "bounded unit cube, 600 Q4 elements (6 x 10 x 10), 64 spheres r=0.05, 32^3 grid",
           "runs": runs, "e2e_includes": "host arrays in, X and 32,768 stresses out (ibem_e3d_run_host)",
           "reference_in_build_container": {
               "value": ref_total, "unit": "s", "layout": 78, "cores": 8, "kind": "reference",
               "sample": ("the reference compiled from its sources (g++ -O2 -fopenmp), 8 x86 threads, when the fixture "
                          f"was made: assembly {asm:.0f} s, fullPivLu {ref['solve']:.0f} s, stresses at 1,024 points "
                          f"{ref['getFlux']:.0f} s scaled to 32,768"), "stages_s": ref}}
    if not args.no_cube64_cpu:
        out["cpu_baseline_24"] = cube64_cpu(c)
    return out


def run_ellipsoids(args, dev):
    """Ellipsoidal inclusions in the dense mixed form (FP32 LU with split-BF16 tensor-core
    updates, FP64 GMRES-IR): args.ellipsoids prolate/oblate ellipsoids, a1 = 0.008,
    a2 = a1 U[0.5, 1], a3 = a1 U[0.25, 1], Haar-uniform orientations, random sequential
    addition with the surfaces kept ~0.2 a3 apart, vf 15%, linear eigenstrain, remote
    sigma33 = 1, stresses on a 16^3 grid.  One step = FP64 pair blocks + right-hand side +
    solve + stresses with inputs in HBM.  The plain FP64 form is timed on args.ell_plain
    ellipsoids of the same distribution (both forms), for the time-to-solution ratio."""
    import torch
    import ibemproject_gb300 as g
    from ibemproject_gb300 import cases
    L = g.lib()
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    out = {}

    def solve_case(num, form, reps):
        c = cases.ellipsoid_case(num, vf=0.15, seed=3, grid=16)
        N = 24 * num
        m = g.material(c.E0, c.nu0, c.E1, c.nu1)
        dv = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)
        cen, ax, qt, pts = dv(c.centers), dv(c.axes), dv(c.quats), dv(c.points)
        A = torch.empty((N, N), dtype=torch.float64, device=dev)
        b = torch.empty(N, dtype=torch.float64, device=dev)
        x = torch.empty_like(b)
        S = torch.empty((c.nump, 6), dtype=torch.float64, device=dev)
        sig = np.ascontiguousarray(c.sig_inf)
        sp = sig.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
        rep = g.SolveReport()
        st = {}
        for it in range(reps):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
            torch.cuda.synchronize()
            ev[0].record()
            g.check(L.ibem_e3d_ell_pair_blocks(P(cen), P(ax), P(qt), num, ctypes.byref(m), P(A), N, 0, 0, None))
            g.check(L.ibem_e3d_farfield_rhs(num, ctypes.byref(m), 24, sp, P(b), None))
            ev[1].record()
            g.check(L.ibem_e3d_solve(form, N, P(A), N, P(b), P(x), 1e-12, ctypes.byref(rep), None))
            ev[2].record()
            g.check(L.ibem_e3d_ell_field(form, P(pts), c.nump, P(cen), P(ax), P(qt), num, ctypes.byref(m), P(x), sp,
                                         P(S), None))
            ev[3].record()
            torch.cuda.synchronize()
            st = {"time_to_solution_s": ev[0].elapsed_time(ev[3]) / 1e3,
                  "stages_ms": {"assembly_rhs": ev[0].elapsed_time(ev[1]), "solve": ev[1].elapsed_time(ev[2]),
                                "field": ev[2].elapsed_time(ev[3])},
                  "backward_error": rep.backward_error, "gmres_iterations": rep.iterations, "N": N,
                  "points": c.nump, "side": float(c.title.split("=")[1])}
        res = (x.cpu().numpy(), S.cpu().numpy())
        del A
        torch.cuda.empty_cache()
        return st, res

    mixed, _ = solve_case(args.ellipsoids, g.SOLVE_MIXED_IR, 2)
    out["mixed_ir"] = mixed
    if args.ell_plain > 0:
        pm, (xm, sm) = solve_case(args.ell_plain, g.SOLVE_MIXED_IR, 2)
        pf, (xf, sf) = solve_case(args.ell_plain, g.SOLVE_FP64, 1)
        pm["rel_err_eigenstrain_vs_fp64"] = float(np.abs(xm - xf).max() / np.abs(xf).max())
        pm["rel_err_stress_vs_fp64"] = float(np.abs(sm - sf).max() / np.abs(sf).max())
        out[f"same_distribution_{args.ell_plain}"] = {"mixed_ir": pm, "plain_fp64": pf,
                                                      "speedup": pf["time_to_solution_s"] / pm["time_to_solution_s"]}
    out["workload"] = (f"{args.ellipsoids} ellipsoids a1=0.008, a2=a1 U[0.5,1], a3=a1 U[0.25,1], Haar orientations, "
                       "RSA, vf 15%, linear eigenstrain (24/particle), far-field sigma33, 16^3 grid")
    return out


def run_ours(args, rank, world):
    import torch
    import ibemproject_gb300 as g
    dev = torch.device("cuda", int(os.environ.get("LOCAL_RANK", 0)))
    torch.cuda.set_device(dev)
    L = g.lib()
    case = make_case(args.num, args.grid, 2024 + rank)   # replicas: one realisation per rank
    N, num, nump = 24 * case.num, case.num, case.nump
    m = g.material(case.E0, case.nu0, case.E1, case.nu1)
    cen = torch.from_numpy(np.ascontiguousarray(case.centers)).to(dev)
    rad = torch.from_numpy(np.ascontiguousarray(case.radius)).to(dev)
    pts = torch.from_numpy(np.ascontiguousarray(case.points)).to(dev)
    b = torch.empty(N, dtype=torch.float64, device=dev)
    x = torch.empty(N, dtype=torch.float64, device=dev)
    S = torch.empty((nump, 6), dtype=torch.float64, device=dev)
    sig = np.ascontiguousarray(case.sig_inf)
    sigp = sig.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    stream = torch.cuda.current_stream(dev)
    sp = ctypes.c_void_p(stream.cuda_stream)
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    rep = g.SolveReport()
    mrep = (g.MfReport * 1)()
    seg = np.array([0, num], dtype=np.int32)
    mats = (g.Material * 1)(m)
    batch = g.Batch(1, seg.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), cen.data_ptr(), rad.data_ptr(), mats)
    opt = g.MfOptions(50, 20, 8, 1e-10, 1e-5)
    params, train_info = (None, None)
    if args.form == "learned_gmres":
        params, train_info = train_preconditioner(args, rank, dev)
    A = None

    def step(form, xo=x, So=S):
        nonlocal A
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
        ev[0].record(stream)
        if form == "learned_gmres":
            g.check(L.ibem_e3d_farfield_rhs(num, ctypes.byref(m), 24, sigp, P(b), sp))
            ev[1].record(stream)
            g.check(L.ibem_e3d_mf_solve(ctypes.byref(batch), P(b), P(xo), g.PRECOND_LEARNED, P(params),
                                        ctypes.byref(opt), mrep, sp))
        else:
            if A is None:
                A = torch.empty((N, N), dtype=torch.float64, device=dev)   # column-major N x N
            f = g.SOLVE_MIXED_IR if form == "mixed_ir" else g.SOLVE_FP64
            g.check(L.ibem_e3d_pair_blocks(P(cen), P(rad), num, ctypes.byref(m), 24, P(A), N, 0, 0, sp))
            g.check(L.ibem_e3d_farfield_rhs(num, ctypes.byref(m), 24, sigp, P(b), sp))
            ev[1].record(stream)
            g.check(L.ibem_e3d_solve(f, N, P(A), N, P(b), P(xo), args.tol, ctypes.byref(rep), sp))
        ev[2].record(stream)
        ff = g.SOLVE_FP64 if form == "plain_fp64" else g.SOLVE_MIXED_IR
        g.check(L.ibem_e3d_field_form(ff, P(pts), nump, P(cen), P(rad), num, ctypes.byref(m), 24, P(xo), None, 0,
                                      None, 0, None, None, sigp, P(So), sp))
        ev[3].record(stream)
        return ev

    def barrier():
        if world > 1:
            torch.distributed.barrier()

    def stages(evs):
        return {"rhs_or_assembly": statistics.median(e[0].elapsed_time(e[1]) for e in evs),
                "solve": statistics.median(e[1].elapsed_time(e[2]) for e in evs),
                "field": statistics.median(e[2].elapsed_time(e[3]) for e in evs)}

    form = args.form
    for _ in range(args.warmup):
        step(form)
    torch.cuda.synchronize()
    barrier()
    clocks = Clocks(dev.index)
    clocks.start()
    launches0 = L.ibem_kernel_launches()
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    t0.record(stream)
    evs = []
    torch.cuda.nvtx.range_push("timed_steps")   # lets ncu select exactly these launches
    for _ in range(args.steps):
        evs.append(step(form))
    torch.cuda.nvtx.range_pop()
    t1.record(stream)
    torch.cuda.synchronize()
    barrier()
    launches = L.ibem_kernel_launches() - launches0
    ck = clocks.stop()
    ms = t0.elapsed_time(t1) / args.steps
    stage_ms = stages(evs)
    solve_info = ({"rel_residual": mrep[0].rel_residual, "refinement_steps": mrep[0].outer,
                   "arnoldi_steps": mrep[0].inner, "setup_ms": mrep[0].t_setup_ms}
                  if form == "learned_gmres" else
                  {"backward_error": rep.backward_error, "gmres_iterations": rep.iterations,
                   "factor_ms": rep.t_factor_ms, "refine_ms": rep.t_solve_ms})
    # one more step with the per-phase CUDA events of the library (kept out of the timed
    # steps above, whose total they would inflate by their own records)
    L.ibem_prof_enable(1)
    step(form)
    torch.cuda.synchronize()
    prof = g.prof_report()
    L.ibem_prof_enable(0)
    ms = job_seconds_per_solution(ms, world, dev) * 1e3

    # the other forms once on the same microstructure, and the chosen form's difference to
    # the plain FP64 solution
    others, prof_mixed = {}, None
    if not args.no_plain and rank == 0:
        x2 = torch.empty(N, dtype=torch.float64, device=dev)
        S2 = torch.empty((nump, 6), dtype=torch.float64, device=dev)
        for f in (["mixed_ir"] if form != "mixed_ir" else []) + ["plain_fp64"]:
            if f == "mixed_ir":
                step(f, x2, S2)   # warm-up of the dense path
                L.ibem_prof_enable(1)
            torch.cuda.synchronize()
            ev = step(f, x2, S2)
            torch.cuda.synchronize()
            if f == "mixed_ir":
                prof_mixed = g.prof_report()
                L.ibem_prof_enable(0)
            others[f] = {"time_to_solution_s": ev[0].elapsed_time(ev[3]) / 1e3, "stages_ms": stages([ev]),
                         "factor_ms": rep.t_factor_ms, "backward_error": rep.backward_error}
            if f == "plain_fp64":
                others[f]["chosen_rel_err_eigenstrain"] = float((x - x2).abs().max() / x2.abs().max())
                others[f]["chosen_rel_err_stress"] = float((S - S2).abs().max() / S2.abs().max())
        del x2, S2
    if form == "mixed_ir":
        prof_mixed = prof
    A = None
    torch.cuda.empty_cache()
    batched = None
    if rank == 0 and args.batch > 0 and params is not None:
        try:
            batched = run_batched(args, dev, params)
        except Exception as ex:   # reported in the JSON line; the headline measurement stands
            batched = {"error": f"{type(ex).__name__}: {ex}"}
        torch.cuda.empty_cache()

    extra = {}
    if rank == 0 and not args.no_cube64:
        try:
            extra["bounded_cube_64_spheres"] = run_cube64(args, dev)
        except Exception as ex:   # reported in the JSON line; the headline measurement stands
            extra["bounded_cube_64_spheres"] = {"error": f"{type(ex).__name__}: {ex}"}
        torch.cuda.empty_cache()
    if rank == 0 and args.large > 0 and params is not None:
        try:
            extra["learned_vs_block_jacobi_large"] = run_large(args, dev, params)
        except Exception as ex:
            extra["learned_vs_block_jacobi_large"] = {"error": f"{type(ex).__name__}: {ex}"}
        torch.cuda.empty_cache()
    if rank == 0 and args.ellipsoids > 0:
        try:
            extra["ellipsoids_mixed"] = run_ellipsoids(args, dev)
        except Exception as ex:
            extra["ellipsoids_mixed"] = {"error": f"{type(ex).__name__}: {ex}"}
        torch.cuda.empty_cache()

    # end to end through the host-buffer C ABI (copies inside the timed region)
    e2e = None
    if rank == 0 and args.e2e_steps > 0:
        hp = params.cpu().numpy() if params is not None else None
        run = (lambda: g.run_host_mf(case, g.PRECOND_LEARNED, hp)) if form == "learned_gmres" else \
              (lambda: g.run_host(case, layout=24, form=g.SOLVE_MIXED_IR, tol=args.tol))
        run()
        t = time.perf_counter()
        for _ in range(args.e2e_steps):
            run()
        e2e_s = (time.perf_counter() - t) / args.e2e_steps
        h2d = case.centers.nbytes + case.radius.nbytes + case.points.nbytes + 48 + (hp.nbytes if hp is not None else 0)
        d2h = 8 * N + 8 * 6 * nump
        e2e = {"value": e2e_s, "unit": "s", "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h)}
    return (case, ms, stage_ms, solve_info, others, e2e, ck, launches, prof, prof_mixed, train_info, batched, extra)


def config_of(args, case, world=1):
    learned = args.form == "learned_gmres"
    return {"workload": WORKLOAD, "layout": 24, "N": 24 * case.num, "points": case.nump, "form": args.form,
            "tol": "relative residual 1e-10 (scaled system)" if learned else f"scaled backward error {args.tol}",
            "l2": ("inputs in HBM; the matrix is never stored (18.4 GB in FP64 if it were)" if learned
                   else "inputs larger than L2 (A is 18.4 GB FP64)"),
            "parallelism": f"replicas x{world}"}


def main():
    args = parse()
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    if args.impl == "reference":
        if rank != 0:
            return 0
        case = make_case(args.num, args.grid, 2024)
        lu = lu_calibration(case)   # timed once; the steps repeat the pair-block and field samples
        for _ in range(max(0, min(args.warmup, 1))):
            cpu_baseline(case, lu=lu)
        vals, cb = [], None
        for _ in range(max(1, args.steps)):
            cb = cpu_baseline(case, lu=lu)
            vals.append(cb["value"])
        v = statistics.median(vals)
        cb["value"] = v
        cb["steps_values"] = vals
        line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "s", "n_gpus": args.gpus,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": v * 1e3, "higher_is_better": False,
                "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded RSA microstructure)",
                "config": config_of(args, case), "cpu_baseline": cb,
                "e2e": {"value": v, "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line))
        return 0

    import torch
    if world > 1:
        torch.distributed.init_process_group("nccl")
    (case, ms, stage_ms, solve_info, others, e2e, ck, launches, prof, prof_mixed,
     train_info, batched, extra) = run_ours(args, rank, world)
    if rank == 0:
        cb = cpu_baseline(case) if world == 1 else None
        N = 24 * case.num
        learned = args.form == "learned_gmres"
        line = {
            "metric": METRIC, "value": ms / 1e3, "unit": "s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None,
            "dtype": "f32 GMRES + f64 refinement" if learned else "f64+f32/bf16x3",
            "data": "synthetic (seeded RSA microstructure)",
            "config": config_of(args, case, world),
            "stages_ms": stage_ms,
            "solve": solve_info,
            "preconditioner_training": train_info,
            "batched_realisations": batched,
            **extra,
            "other_forms": others,
            "e2e": e2e,
            "clocks": ck,
            "gpu_launches": int(launches),
            "profile_ms_per_step": {k: {"launches": v["launches"], "ms": v["ms"]} for k, v in prof.items()},
            "profile_note": "one extra step after the timed ones, with CUDA events around each phase",
            "roofline": roofline_chosen(prof, case) if learned else roofline(prof),
            "roofline_tensor_gemm": roofline(prof_mixed) if prof_mixed else None,
            "cpu_baseline": cb,
        }
        print(json.dumps(line))
    if world > 1:
        torch.distributed.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
