#!/usr/bin/env python
"""Time-to-solution benchmark of the ripley/paso hot path on B200.

Workload (one step = one pass of the hot path over one synthetic input): ripley Brick
128^3 Q1 elements on [0,1]^3, A = kappa*I with kappa = exp(g), g a Gaussian random field
(white noise smoothed with a Gaussian of 8 cells, standardised, periodic), Y = sum of 4
Gaussian blobs (width 3 cells, amplitudes U(-1,1), centres uniform) at the Gauss points,
u = 0 on the top face z = 1, PCG + Jacobi to relative residual 1e-8.  A step is: reset
the matrix, assemble A and Y, insert the Dirichlet constraint, solve.  The timed path is
the FP32-inner / FP64-refinement PCG on the band layout; the plain FP64 paso PCG on the
CSR matrix (the reference algorithm) is timed beside it on the same input.

Usage (driver contract):
  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
N>1 runs as one process per GPU under torch.distributed.run; every rank solves its
own independent instance (weak scaling, no collective on the data path).
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

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
PKG_DIR = os.path.join(REPO, "esys-escript.github.io_b200")
for p in (PKG_DIR, REPO):
    if p not in sys.path:
        sys.path.insert(0, p)

METRIC = "time-to-1e-8 residual, Brick 128^3: learned+FP32 refine vs plain FP64 PCG, B200"
RTOL = 1e-8


# ----------------------------------------------------------------------------------------------
# synthetic inputs (seeded)
# ----------------------------------------------------------------------------------------------

def make_inputs(ne: int, seed: int, corr_cells: float):
    """kappa per element (element order k0 + NE k1 + NE^2 k2), Y at the Gauss points
    (NE^3 x 8, q x-fastest) and the Dirichlet mask of the top face."""
    from scipy.ndimage import gaussian_filter
    rng = np.random.default_rng(seed)
    g = gaussian_filter(rng.standard_normal((ne, ne, ne)), sigma=corr_cells, mode="wrap")
    g = (g - g.mean()) / g.std()
    kappa = np.exp(g).reshape(-1)
    h = 1.0 / ne
    gp = np.array([0.5 - np.sqrt(3) / 6, 0.5 + np.sqrt(3) / 6])
    axis = (np.arange(ne)[:, None] + gp[None, :]) * h  # (NE, 2) Gauss coordinates
    amps = rng.uniform(-1.0, 1.0, 4)
    centres = rng.uniform(0.0, 1.0, (4, 3))
    w = 3.0 * h
    Y = np.zeros((ne, ne, ne, 2, 2, 2))  # (k2, k1, k0, qz, qy, qx)
    for a, c in zip(amps, centres):
        f = [np.exp(-((axis - c[d]) ** 2) / (2 * w * w)) for d in range(3)]
        Y += a * (f[2][:, None, None, :, None, None] * f[1][None, :, None, None, :, None] *
                  f[0][None, None, :, None, None, :])
    nn = ne + 1
    q = np.zeros(nn ** 3)
    q[(nn - 1) * nn * nn:] = 1.0
    return {"kappa": kappa, "Y": Y.reshape(-1), "q": q, "ne": ne, "seed": seed,
            "amps": amps.tolist(), "centres": centres.tolist()}


# ----------------------------------------------------------------------------------------------
# clocks during the timed region
# ----------------------------------------------------------------------------------------------

class ClockSampler:
    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_id: str | None):
        self.gpu_id = gpu_id
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        cmd = ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits", "-lms", "200"]
        if self.gpu_id:
            cmd += ["-i", self.gpu_id]
        try:
            self.proc = subprocess.Popen(cmd, stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 8:
                rows.append(parts)
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[0]) for r in rows if r[0].replace(".", "").isdigit()]
        mx = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({n for r in rows for n, v in zip(names, r[4:8]) if v.lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


# ----------------------------------------------------------------------------------------------
# CPU baseline: the reference's own assembler + paso solver (oracle/_ref), else the oracle port
# ----------------------------------------------------------------------------------------------

def _reference_system(inp, use_ref):
    """The reference's assembly (DefaultAssembler3D with A expanded to the Gauss points, the
    form escript hands it) and insertConstraint of the full input.  Returns the pattern,
    values, right hand side and the two times."""
    from oracle import oracle as O
    ne = inp["ne"]
    nel = ne ** 3
    A = np.zeros((nel, 8, 3, 3))
    for i in range(3):
        A[:, :, i, i] = inp["kappa"][:, None]
    A = A.reshape(-1)
    pat = O.pattern(3, (ne, ne, ne))
    t0 = time.perf_counter()
    val, rhs = O.assemble(3, (ne, ne, ne), [1.0 / ne] * 3, pat, A=(O.EXPANDED, A),
                          Y=(O.EXPANDED, inp["Y"]), use_ref=use_ref)
    t1 = time.perf_counter()
    O.insert_constraint(pat, val, rhs, inp["q"])
    t2 = time.perf_counter()
    return pat, val, rhs, t1 - t0, t2 - t1


def cpu_reference_solve(inp, threads, rtol=RTOL, oracle_rtol=None):
    """One complete time-to-solution of the reference on the host cores: its own assembly,
    the constraint and paso's Solver/PCG to rtol (oracle/_ref, the reference's sources
    compiled in place; the oracle port where that library is absent).  With oracle_rtol it
    also solves the same system to that tolerance (untimed) and returns that solution as
    the FP64 oracle the GPU solutions are measured against."""
    from oracle import oracle as O
    use_ref = O.have_ref()
    kind = "reference" if use_ref else "port"
    if use_ref:
        O.set_threads(threads)
    else:
        os.environ["OMP_NUM_THREADS"] = str(threads)
    pat, val, rhs, t_asm, t_con = _reference_system(inp, use_ref)
    val0 = val.copy() if oracle_rtol else None
    s0 = time.perf_counter()
    r = O.solve_paso(pat, val, rhs, tol=rtol, use_ref=use_ref)
    t_sol = time.perf_counter() - s0
    out = {"kind": kind, "cores": threads, "assemble_s": t_asm, "constraint_s": t_con, "solve_s": t_sol,
           "time_to_solution_s": t_asm + t_con + t_sol, "iterations": int(r.num_iter),
           "converged": bool(r.converged), "x": r.x}
    if oracle_rtol:
        ro = O.solve_paso(pat, val0, rhs, tol=oracle_rtol, use_ref=use_ref)
        out["x_oracle"] = ro.x
        out["oracle_iterations"] = int(ro.num_iter)
    return out


def cpu_reference_warmup(inp, threads):
    """A bounded warm-up of the reference on the host: assembly, constraint and 10 paso
    iterations (pages the code and the arrays in)."""
    from oracle import oracle as O
    use_ref = O.have_ref()
    if use_ref:
        O.set_threads(threads)
    pat, val, rhs, _, _ = _reference_system(inp, use_ref)
    O.solve_paso(pat, val, rhs, tol=RTOL, iter_max=10, use_ref=use_ref)


# ----------------------------------------------------------------------------------------------
# our arm
# ----------------------------------------------------------------------------------------------

# algorithmic bytes per iteration of the dominant kernel, per DOF (n); a launch runs many
# iterations.  One FP32 PCG iteration reads the row's operator data and its 16-byte iteration
# state {u, D^-1 A u, D^-1 A p, p}, writes the new state, and updates the correction d (read +
# write: every iteration on the band copy, every second one on the element coefficients).
# Operator data: the element coefficient of the row's node (4 B, RG_LAYOUT_COEF, the timed
# path), or the row's 27 band values (4 B each, padded bands count, RG_LAYOUT_BAND)
F32_COEF_BYTES_PER_ROW = 4 + 16 + 16 + 4
F32_SPMV_BYTES_PER_ROW = 27 * 4 + 16 + 16 + 8


def max_over_ranks_of(v, dist=None, device="cpu"):
    """The largest of every rank's v (the whole job's time); v itself on one process."""
    if dist is None:
        return v
    import torch
    t = torch.tensor([float(v)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def run_ours(args):
    import ctypes as C
    import torch
    from esys_b200 import _lib as L

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300),
                                device_id=torch.device("cuda", local))
    lib = L.lib()
    ne = args.ne
    inp = make_inputs(ne, args.seed + rank, 8.0 * ne / 128.0)
    nel = ne ** 3
    dev = torch.device("cuda", local)
    stream = torch.cuda.current_stream()
    L.set_stream_from_torch()

    # device-resident inputs: A per element (kappa*I, 9 values), Y at the Gauss points, q
    A_pe = np.zeros((nel, 3, 3))
    for i in range(3):
        A_pe[:, i, i] = inp["kappa"]
    A_host = torch.from_numpy(A_pe.reshape(-1)).pin_memory()
    Y_host = torch.from_numpy(inp["Y"]).pin_memory()
    q_host = torch.from_numpy(inp["q"]).pin_memory()
    A_d = A_host.to(dev)
    Y_d = Y_host.to(dev)
    q_d = q_host.to(dev)

    dom = C.c_void_p()
    ne3 = (C.c_int64 * 3)(ne, ne, ne)
    L.check(lib.rg_domain_create(3, ne3, (C.c_double * 3)(0, 0, 0), (C.c_double * 3)(1, 1, 1), C.byref(dom)))
    n, nnz = C.c_int64(), C.c_int64()
    L.check(lib.rg_domain_info(dom, C.byref(n), C.byref(nnz), None, None, None))
    n, nnz = n.value, nnz.value
    mat = C.c_void_p()
    L.check(lib.rg_matrix_create(dom, C.byref(mat)))
    if args.spmv_config >= 0:  # profiling runs: a fixed FP32 SpMV pipeline instead of the tuner's
        L.check(lib.rg_solver_set_config(mat, args.spmv_config))
    rhs = torch.zeros(n, dtype=torch.float64, device=dev)
    x = torch.zeros(n, dtype=torch.float64, device=dev)

    rtol = args.rtol

    def opts(mode, precision, tol=None):
        tol = rtol if tol is None else tol
        o = L.rg_solver_opts()
        lib.rg_solver_opts_default(C.byref(o))
        o.tolerance = tol
        o.mode = mode
        o.precision = precision
        o.layout = L.RG_LAYOUT_COEF if precision == L.RG_PREC_FP32_REFINE else L.RG_LAYOUT_CSR
        return o

    fast = opts(L.RG_MODE_STANDARD, L.RG_PREC_FP32_REFINE)
    if args.inner == "band":  # profiling runs: the FP32 iterations on the band copy
        fast.layout = L.RG_LAYOUT_BAND
    if args.inner_tol > 0:
        fast.inner_tolerance = args.inner_tol
    plain = opts(L.RG_MODE_PASO, L.RG_PREC_FP64)
    empty = L.rg_coef(None, 0)
    cA = L.rg_coef(A_d.data_ptr(), L.RG_COEF_PER_ELEMENT)
    cY = L.rg_coef(Y_d.data_ptr(), L.RG_COEF_EXPANDED)

    # learned warm start: the network trained on 64^3 solves, applied to the fields coarsened
    # to 64^3 and interpolated to the nodes; Chebyshev-smoothed inside the solver
    from esys_b200 import warmstart as WS
    warm = WS.WarmStart(WS.UNet.load(device=dev))
    guess = torch.zeros(n, dtype=torch.float64, device=dev)
    kap32 = torch.empty((1, ne, ne, ne), dtype=torch.float32, device=dev)
    y32 = torch.empty_like(kap32)
    learned = opts(L.RG_MODE_STANDARD, L.RG_PREC_FP32_REFINE)
    learned.initial_guess = guess.data_ptr()
    if args.inner_tol > 0:
        learned.inner_tolerance = args.inner_tol
    learned.guess_sweeps = args.sweeps
    timed = learned if args.path == "learned" else fast
    side = torch.cuda.Stream(device=dev)

    def step(o, A_dev=None, Y_dev=None, q_dev=None):
        ca = cA if A_dev is None else L.rg_coef(A_dev.data_ptr(), L.RG_COEF_PER_ELEMENT)
        cy = cY if Y_dev is None else L.rg_coef(Y_dev.data_ptr(), L.RG_COEF_EXPANDED)
        qq = q_d if q_dev is None else q_dev
        if o is learned:
            side.wait_stream(stream)  # the inputs are on the main stream
        # the assembly (memory-bound) is queued first on the main stream, so that it runs
        # while the host queues the network's launches on the second stream
        L.set_stream_from_torch()
        L.check(lib.rg_matrix_reset(mat))
        rhs.zero_()
        L.check(lib.rg_assemble_single(mat, C.c_void_p(rhs.data_ptr()), C.byref(ca), C.byref(empty),
                                       C.byref(empty), C.byref(empty), C.byref(empty), C.byref(cy)))
        L.check(lib.rg_insert_constraint(mat, C.c_void_p(rhs.data_ptr()), C.c_void_p(qq.data_ptr()), None, 0))
        if o is learned:
            # the network (tensor-core convolutions) on the second stream; the solve waits for
            # both.  Network input: kappa (A's first diagonal entry) and Y per element
            Ad = A_d if A_dev is None else A_dev
            Yd = Y_d if Y_dev is None else Y_dev
            with torch.cuda.stream(side):
                L.set_stream_from_torch()
                L.check(lib.rg_ws_element_fields(C.c_void_p(Ad.data_ptr()), 9, C.c_void_p(Yd.data_ptr()), 8,
                                                 nel, C.c_void_p(kap32.data_ptr()), C.c_void_p(y32.data_ptr())))
                warm.guess(kap32, y32, (ne, ne, ne), q=qq, out=guess)
            L.set_stream_from_torch()  # library work back on the main stream
        d = L.rg_diag()
        if o is learned:
            stream.wait_stream(side)
        L.check(lib.rg_solve(mat, C.c_void_p(rhs.data_ptr()), C.c_void_p(x.data_ptr()), C.byref(o), C.byref(d)))
        return d

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    def max_over_ranks(v):
        return max_over_ranks_of(v, dist, dev)

    if args.only in ("plain", "plain_band"):
        o = plain
        if args.only == "plain_band":
            o = opts(L.RG_MODE_PASO, L.RG_PREC_FP64)
            o.layout = L.RG_LAYOUT_BAND
        for _ in range(args.warmup + args.steps):
            step(o)
        torch.cuda.synchronize()
        print(json.dumps({"only": args.only, "iterations": int(step(o).num_iter)}), flush=True)
        return
    if args.only == "fast":
        for _ in range(args.warmup):
            d = step(timed)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            d = step(timed)
        e1.record(stream)
        torch.cuda.synchronize()
        # the iteration kernel's time per iteration (events around every launch, one step)
        lib.rg_timers_reset()
        lib.rg_timers_enable(1)
        d = step(timed)
        torch.cuda.synchronize()
        lib.rg_timers_enable(0)
        kms = L.timers()["f32_spmv"][2]
        print(json.dumps({"only": "fast", "path": args.path, "iterations": int(d.num_iter),
                          "outer_steps": int(d.num_outer), "inner_operator": int(d.inner_operator),
                          "fp64_fallback": int(d.fp64_fallback), "ms_per_step": e0.elapsed_time(e1) / args.steps,
                          "iteration_kernel_us": kms / max(int(d.num_iter), 1) * 1e3}), flush=True)
        return

    # --- FP64 reference solution for the error statement (paso algorithm, rtol 1e-10, or
    # 100x below the workload's tolerance when that is tighter)
    step(opts(L.RG_MODE_PASO, L.RG_PREC_FP64, min(1e-10, rtol / 100)))
    x_fp64 = x.clone()

    # --- plain FP64 paso PCG (the reference algorithm) on the same input
    d_plain = step(plain)
    plain_iters = int(d_plain.num_iter)
    barrier()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    n_plain = max(2, min(args.steps, 3))
    ev0.record(stream)
    for _ in range(n_plain):
        d_plain = step(plain)
    ev1.record(stream)
    torch.cuda.synchronize()
    plain_ms = max_over_ranks(ev0.elapsed_time(ev1) / n_plain)
    x_plain = x.clone()

    # --- the same FP64 paso PCG with its SpMV on the FP64 band copy (RG_LAYOUT_BAND)
    plain_band = opts(L.RG_MODE_PASO, L.RG_PREC_FP64)
    plain_band.layout = L.RG_LAYOUT_BAND
    d_pb = step(plain_band)
    barrier()
    ev0.record(stream)
    for _ in range(n_plain):
        d_pb = step(plain_band)
    ev1.record(stream)
    torch.cuda.synchronize()
    plain_band_ms = max_over_ranks(ev0.elapsed_time(ev1) / n_plain)
    x_plain_band = x.clone()

    # --- textbook Jacobi-PCG in FP64 (RG_MODE_STANDARD) on the FP64 band copy: the fastest
    # FP64 solve of the library, the baseline the mixed-precision speed-up is quoted against
    std_band = opts(L.RG_MODE_STANDARD, L.RG_PREC_FP64)
    std_band.layout = L.RG_LAYOUT_BAND
    d_sb = step(std_band)
    barrier()
    ev0.record(stream)
    for _ in range(n_plain):
        d_sb = step(std_band)
    ev1.record(stream)
    torch.cuda.synchronize()
    std_band_ms = max_over_ranks(ev0.elapsed_time(ev1) / n_plain)
    x_std_band = x.clone()

    # --- the FP32-refinement path without the learned guess, for comparison
    for _ in range(2):
        step(fast)
    barrier()
    ev0.record(stream)
    n_f = max(2, min(args.steps, 3))
    for _ in range(n_f):
        d_f32 = step(fast)
    ev1.record(stream)
    torch.cuda.synchronize()
    f32_ms = max_over_ranks(ev0.elapsed_time(ev1) / n_f)
    x_f32 = x.clone()

    # --- the same FP32 refinement with the operator streamed from the FP32 band copy
    # (RG_LAYOUT_BAND) instead of evaluated from the element coefficients
    fast_band = opts(L.RG_MODE_STANDARD, L.RG_PREC_FP32_REFINE)
    fast_band.layout = L.RG_LAYOUT_BAND
    step(fast_band)
    barrier()
    ev0.record(stream)
    for _ in range(n_f):
        d_fb = step(fast_band)
    ev1.record(stream)
    torch.cuda.synchronize()
    f32_band_ms = max_over_ranks(ev0.elapsed_time(ev1) / n_f)
    x_f32_band = x.clone()
    # its iteration kernel's time per iteration (events around every launch, one step)
    lib.rg_timers_reset()
    lib.rg_timers_enable(1)
    d_fb = step(fast_band)
    torch.cuda.synchronize()
    lib.rg_timers_enable(0)
    band_us = L.timers()["f32_spmv"][2] / max(int(d_fb.num_iter), 1) * 1e3

    # --- the same with A given expanded (its 9 values repeated at the 8 Gauss points, the form
    # escript's general assembler reads): the assembly reads 1.2 GB of A instead of 151 MB
    A_x = A_d.view(-1, 1, 9).expand(-1, 8, 9).contiguous()
    cAx = L.rg_coef(A_x.data_ptr(), L.RG_COEF_EXPANDED)

    def step_expanded():
        L.check(lib.rg_matrix_reset(mat))
        rhs.zero_()
        L.check(lib.rg_assemble_single(mat, C.c_void_p(rhs.data_ptr()), C.byref(cAx), C.byref(empty),
                                       C.byref(empty), C.byref(empty), C.byref(empty), C.byref(cY)))
        L.check(lib.rg_insert_constraint(mat, C.c_void_p(rhs.data_ptr()), C.c_void_p(q_d.data_ptr()), None, 0))
        d = L.rg_diag()
        L.check(lib.rg_solve(mat, C.c_void_p(rhs.data_ptr()), C.c_void_p(x.data_ptr()), C.byref(fast), C.byref(d)))
        return d

    step_expanded()
    barrier()
    ev0.record(stream)
    for _ in range(n_f):
        d_fx = step_expanded()
    ev1.record(stream)
    torch.cuda.synchronize()
    f32x_ms = max_over_ranks(ev0.elapsed_time(ev1) / n_f)
    A_x_host = A_x.cpu().pin_memory()

    # --- warm-up of the timed path
    for _ in range(args.warmup):
        step(timed)
    barrier()

    # --- timed region: K steps of the fast path
    gpu_id = None
    try:
        gpu_id = "GPU-" + str(torch.cuda.get_device_properties(local).uuid)
    except Exception:
        gpu_id = None
    clocks = ClockSampler(gpu_id)
    lib.rg_timers_reset()
    clocks.start()
    barrier()
    ev0.record(stream)
    for _ in range(args.steps):
        d_fast = step(timed)
    ev1.record(stream)
    torch.cuda.synchronize()
    clk = clocks.stop()
    ms = max_over_ranks(ev0.elapsed_time(ev1) / args.steps)
    launches = int(sum(v[0] for v in L.timers().values()))
    x_fast = x.clone()
    err = float((x_fast - x_fp64).norm() / x_fp64.norm())

    # --- kernel timing: the same steps with CUDA events around every library launch (on the
    # launching stream)
    n_prof = max(1, min(args.steps, 3))
    lib.rg_timers_reset()
    lib.rg_timers_enable(1)
    barrier()
    ev0.record(stream)
    prof_iters = 0
    for _ in range(n_prof):
        prof_iters += int(step(timed).num_iter)
    ev1.record(stream)
    torch.cuda.synchronize()
    lib.rg_timers_enable(0)
    ms_events = ev0.elapsed_time(ev1) / n_prof
    tm = L.timers()

    # dominant kernel: the FP32 iterations; time per iteration from the live events (the passes
    # that start a segment included)
    spmv_n, spmv_t, spmv_ms = tm["f32_spmv"]
    avg_s = spmv_ms / max(prof_iters, 1) / 1e3
    coef_used = bool(d_fast.inner_operator)
    algo_bytes = (F32_COEF_BYTES_PER_ROW if coef_used else F32_SPMV_BYTES_PER_ROW) * n
    peaks = {}
    pk_path = os.path.join(REPO, "MEASURED_PEAKS.json")
    if os.path.exists(pk_path):
        peaks = json.load(open(pk_path))
    hbm = peaks.get("hbm_gbs")
    peak_note = "of measured" if hbm else "of fallback"
    hbm = hbm or 6650.0
    achieved = algo_bytes / avg_s / 1e9 if avg_s > 0 else 0.0
    # DRAM bytes per iteration of the same kernel from one ncu capture (profiles/traffic.json)
    tr_all = {}
    tr_path = os.path.join(REPO, "profiles", "traffic.json")
    if os.path.exists(tr_path):
        tr_all = {k: v for k, v in json.load(open(tr_path)).items() if v.get("ne") == ne}
    tr = tr_all.get("f32_cg_coef" if coef_used else "f32_cg_band", {})
    traffic, limiter = tr.get("bytes_per_iteration"), tr.get("limiter")
    roofline = {"bound": "hbm",
                "kernel": ("k_f32_cg_coef<3> (FP32 PCG iterations, many per launch: operator from kappa per "
                           "element, vector updates, one grid-wide exchange each)" if coef_used else
                           "k_f32_cg<27> (FP32 PCG iterations, many per launch: 27-band SpMV, vector updates, one "
                           "grid-wide exchange each)"),
                "achieved": round(achieved, 1), "peak": hbm, "unit": "GB/s",
                "frac": round(achieved / hbm, 4), "peak_source": peak_note,
                "algorithmic_bytes_per_iteration": algo_bytes, "avg_iteration_us": round(avg_s * 1e6, 2),
                "iterations_timed": prof_iters, "launches_timed": spmv_t, "traffic": traffic, "limiter": limiter,
                "timing": f"CUDA events around each launch over {n_prof} steps ({ms_events:.1f} ms/step)"}

    # the pipeline configuration the tuner chose for the timed path's operator (read before
    # another solve switches the matrix's workspace to another operator)
    cfg, ug = C.c_int(), C.c_int()
    spmv_us = (C.c_double * 2)()
    lib.rg_solver_config(mat, C.byref(cfg), C.byref(ug), spmv_us)
    spmv_names = ({0: "k_f32_cg_coef<3, 2 lines/warp, 16 warps/CTA>",
                   1: "k_f32_cg_coef<3, 1 line/warp, 28 warps/CTA>"} if coef_used else
                  {0: "k_f32_cg<27, 3 stages x 1 CTA/SM>", 1: "k_f32_cg<27, 2 stages x 2 CTAs/SM>"})
    roofline["kernel"] = spmv_names.get(cfg.value, roofline["kernel"])
    roofline["tuned"] = {"spmv_config": cfg.value, "update_grid": ug.value,
                         "spmv_us_per_config": [round(v, 2) for v in spmv_us]}

    # --- textbook FP64 PCG on the same input (information: iteration count of CG without smoothing)
    d_std = step(opts(L.RG_MODE_STANDARD, L.RG_PREC_FP64))

    # --- end to end through the C-ABI with host buffers (pinned), copies inside the timed region
    bi = A_host.numel() * 8 + Y_host.numel() * 8 + q_host.numel() * 8
    bo = n * 8
    x_host = torch.empty(n, dtype=torch.float64).pin_memory()
    A_e = torch.empty_like(A_d)
    Y_e = torch.empty_like(Y_d)
    q_e = torch.empty_like(q_d)
    barrier()
    ev0.record(stream)
    for _ in range(args.steps):
        A_e.copy_(A_host, non_blocking=True)
        Y_e.copy_(Y_host, non_blocking=True)
        q_e.copy_(q_host, non_blocking=True)
        step(timed, A_e, Y_e, q_e)
        x_host.copy_(x, non_blocking=True)
    ev1.record(stream)
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks(ev0.elapsed_time(ev1) / args.steps)

    # --- the same end to end with A handed over the way escript's LinearPDE does when kappa
    # lives on Function: expanded to the 8 Gauss points (72 doubles per element, 1.2 GB at
    # 128^3), copied from pinned host memory every step; the learned path reads kappa from it
    def step_expanded_e2e():
        A_x.copy_(A_x_host, non_blocking=True)
        Y_e.copy_(Y_host, non_blocking=True)
        q_e.copy_(q_host, non_blocking=True)
        cax = L.rg_coef(A_x.data_ptr(), L.RG_COEF_EXPANDED)
        if timed is learned:
            side.wait_stream(stream)
            with torch.cuda.stream(side):
                L.set_stream_from_torch()
                L.check(lib.rg_ws_element_fields(C.c_void_p(A_x.data_ptr()), 72, C.c_void_p(Y_e.data_ptr()), 8,
                                                 nel, C.c_void_p(kap32.data_ptr()), C.c_void_p(y32.data_ptr())))
                warm.guess(kap32, y32, (ne, ne, ne), q=q_e, out=guess)
            L.set_stream_from_torch()
        L.check(lib.rg_matrix_reset(mat))
        rhs.zero_()
        L.check(lib.rg_assemble_single(mat, C.c_void_p(rhs.data_ptr()), C.byref(cax), C.byref(empty),
                                       C.byref(empty), C.byref(empty), C.byref(empty),
                                       C.byref(L.rg_coef(Y_e.data_ptr(), L.RG_COEF_EXPANDED))))
        L.check(lib.rg_insert_constraint(mat, C.c_void_p(rhs.data_ptr()), C.c_void_p(q_e.data_ptr()), None, 0))
        if timed is learned:
            stream.wait_stream(side)
        d = L.rg_diag()
        L.check(lib.rg_solve(mat, C.c_void_p(rhs.data_ptr()), C.c_void_p(x.data_ptr()), C.byref(timed), C.byref(d)))
        x_host.copy_(x, non_blocking=True)
        return d

    step_expanded_e2e()
    barrier()
    n_x = max(2, min(args.steps, 3))
    ev0.record(stream)
    for _ in range(n_x):
        step_expanded_e2e()
    ev1.record(stream)
    torch.cuda.synchronize()
    e2e_x_ms = max_over_ranks(ev0.elapsed_time(ev1) / n_x)
    bi_x = A_x_host.numel() * 8 + Y_host.numel() * 8 + q_host.numel() * 8
    del A_x, A_x_host

    # --- CPU baseline (rank 0, one GPU): the reference's own code on a bounded sample
    cpu = None
    errors = None
    if rank == 0 and world == 1 and not args.no_cpu:
        threads = os.cpu_count() or 1
        oracle_rtol = min(1e-10, rtol / 100)
        s = cpu_reference_solve(inp, threads, rtol=rtol, oracle_rtol=oracle_rtol)
        cpu = {"value": round(s["time_to_solution_s"] * 1e3, 1), "unit": "ms", "cores": threads,
               "kind": s["kind"],
               "sample": (f"one complete time-to-solution of the reference on the full {ne}^3 input: its "
                          f"DefaultAssembler3D (A on the Gauss points) + insertConstraint + paso Solver/PCG "
                          f"to rtol {rtol:g} ({s['iterations']} iterations)"),
               "assemble_s": round(s["assemble_s"], 3), "constraint_s": round(s["constraint_s"], 3),
               "solve_s": round(s["solve_s"], 3), "iterations": s["iterations"]}
        xo = s["x_oracle"]
        nrm = float(np.linalg.norm(xo))

        def err_of(v):
            return float(np.linalg.norm(v.cpu().numpy() - xo) / nrm)

        errors = {"oracle": (f"{s['kind']} paso Solver/PCG in FP64 on the host, rtol {oracle_rtol:g} "
                             f"({s['oracle_iterations']} iterations)"),
                  "timed_path": err_of(x_fast), "fp32_refine_no_guess": err_of(x_f32),
                  "fp32_refine_band": err_of(x_f32_band),
                  "plain_fp64_paso_csr": err_of(x_plain), "plain_fp64_paso_band": err_of(x_plain_band),
                  "fp64_standard_band": err_of(x_std_band),
                  "reference_at_rtol": float(np.linalg.norm(s["x"] - xo) / nrm)}

    kernels = {k: {"launches_per_step": v[0] // n_prof, "ms_per_step": round(v[2] / n_prof, 3)}
               for k, v in tm.items() if v[0]}
    band_bytes = F32_SPMV_BYTES_PER_ROW * n
    roofline_band = {"kernel": "k_f32_cg<27> (the same iterations streaming the FP32 band copy)",
                     "algorithmic_bytes_per_iteration": band_bytes, "avg_iteration_us": round(band_us, 2),
                     "achieved": round(band_bytes / (band_us * 1e-6) / 1e9, 1), "peak": hbm, "unit": "GB/s",
                     "frac": round(band_bytes / (band_us * 1e-6) / 1e9 / hbm, 4), "peak_source": peak_note,
                     "traffic": tr_all.get("f32_cg_band", {}).get("bytes_per_iteration")}

    # --- batched workload: 64 Bricks with edges from {32,48,64,80,96} per axis, 8 right hand
    # sides each, FP32-inner/FP64-refinement PCG to rtol 1e-8, one batch (timed separately)
    batched = None
    if args.batched:
        from esys_b200.batch import BatchSolver, make_batch
        systems, brhs = make_batch(64, 8, seed=args.seed)
        bx = [torch.zeros_like(b) for b in brhs]
        with BatchSolver([sy.mat for sy in systems], 8) as bs:
            info = bs.tune()
            bs.solve(brhs, bx)
            barrier()
            ev0.record(stream)
            bd = bs.solve(brhs, bx)
            ev1.record(stream)
            torch.cuda.synchronize()
            b_ms = max_over_ranks(ev0.elapsed_time(ev1))
        its = [x.num_iter for x in bd]
        unknowns = sum(sy.n for sy in systems) * 8
        batched = {"workload": "64 Bricks, edges uniform from {32,48,64,80,96} per axis, own kappa each "
                               "(corr 8 cells), 8 RHS each (4 Gaussian blobs), rtol 1e-8",
                   "ms": round(b_ms, 2), "unknowns_x_rhs": unknowns,
                   "unknowns_per_s": round(unknowns / (b_ms / 1e3), 1),
                   "all_converged": all(x.converged for x in bd),
                   "iterations": {"min": min(its), "mean": round(float(np.mean(its)), 1), "max": max(its)},
                   "outer_steps": int(bd[0].num_outer), "tuned": info}
        for sy in systems:
            sy.close()
    out = {
        "metric": METRIC, "value": round(ms, 3), "unit": "ms", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms, 3), "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32 inner / f64 refine",
        "data": "synthetic, seeded: kappa=exp(GRF corr 8 cells, std 1), 4 Gaussian blobs",
        "config": {"workload": f"Brick {ne}^3 variable-coefficient Poisson, u=0 on top face, "
                               f"PCG+Jacobi rtol {rtol:g} (assemble+constrain+solve per step)",
                   "ne": [ne, ne, ne], "n_dof": n, "nnz": nnz, "seed": args.seed,
                   "path": ("learned warm start (U-Net on tcgen05, fields coarsened to 64^3, Chebyshev-"
                            f"smoothed x{args.sweeps}) + FP32 PCG (operator from the element coefficients, one "
                            "fused kernel per iteration) with FP64 residual replacement"
                            if args.path == "learned" else
                            "FP32 PCG (operator from the element coefficients, one fused kernel per iteration) with "
                            "FP64 residual replacement"),
                   "l2": (f"inputs larger than L2 (FP64 CSR values {nnz * 8 / 1e6:.0f} MB, band copy "
                          f"{27 * 4 * n / 1e6:.0f} MB per step)"),
                   "parallelism": f"{world} independent replicas" if world > 1 else "1 GPU"},
        "iterations": int(d_fast.num_iter), "outer_steps": int(d_fast.num_outer),
        "rel_residual": float(d_fast.residual_norm / d_fast.rhs_norm),
        "error_vs_fp64": err,
        "error_vs_oracle": errors["timed_path"] if errors else None,
        "errors_vs_oracle": errors,
        "inner_operator": "element coefficients" if coef_used else "band copy",
        "plain_fp64": {"ms": round(plain_ms, 3), "iterations": plain_iters,
                       "algorithm": "paso PCG with residual smoothing, balanced CSR FP64",
                       "band_layout_ms": round(plain_band_ms, 3),
                       "band_layout_iterations": int(d_pb.num_iter),
                       "standard_band_ms": round(std_band_ms, 3),
                       "standard_band_iterations": int(d_sb.num_iter),
                       "fastest_ms": round(min(plain_ms, plain_band_ms, std_band_ms), 3)},
        "speedup_vs_plain_fp64": round(min(plain_ms, plain_band_ms, std_band_ms) / ms, 3),
        "speedup_vs_paso_csr": round(plain_ms / ms, 3),
        "fp32_refine_no_guess": {"ms": round(f32_ms, 3), "iterations": int(d_f32.num_iter),
                                 "inner_operator": "element coefficients" if d_f32.inner_operator else "band copy",
                                 "speedup_vs_plain_fp64": round(min(plain_ms, plain_band_ms, std_band_ms) / f32_ms, 3),
                                 "with_A_expanded_ms": round(f32x_ms, 3),
                                 "with_A_expanded_iterations": int(d_fx.num_iter)},
        "fp32_refine_band": {"ms": round(f32_band_ms, 3), "iterations": int(d_fb.num_iter),
                             "inner_operator": "band copy (RG_LAYOUT_BAND)", "roofline": roofline_band},
        "learned_guess": ({"rejected": bool(d_fast.guess_rejected),
                           "guess_rel_residual": float(d_fast.guess_residual / d_fast.rhs_norm),
                           "smoothing_steps": args.sweeps,
                           "iterations_saved": int(d_f32.num_iter) - int(d_fast.num_iter),
                           "weights": "esys_b200/data/warmstart_unet.npz (20k 64^3 solves, val rel l2 0.29)"}
                          if args.path == "learned" else None),
        "std_fp64_iterations": int(d_std.num_iter),
        "roofline": roofline, "cpu_baseline": cpu,
        "e2e": {"value": round(e2e_ms, 3), "unit": "ms", "h2d_bytes_per_step": bi, "d2h_bytes_per_step": bo},
        "e2e_A_expanded": {"value": round(e2e_x_ms, 3), "unit": "ms", "h2d_bytes_per_step": bi_x,
                           "d2h_bytes_per_step": bo,
                           "note": "A as escript hands it for kappa on Function: 72 doubles per element"},
        "gpu_launches": launches, "clocks": clk, "kernels": kernels,
        "batched": batched,
    }
    lib.rg_matrix_destroy(mat)
    lib.rg_domain_destroy(dom)
    if rank == 0:
        print(json.dumps(out), flush=True)
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()


# ----------------------------------------------------------------------------------------------
# reference arm: the reference's own CPU implementation of the path on the host cores
# ----------------------------------------------------------------------------------------------

def run_reference(args):
    """The reference's own CPU implementation of the path on the host cores: every timed step
    is one complete time-to-solution of the same workload (DefaultAssembler3D with A on the
    Gauss points, insertConstraint, paso Solver/PCG to rtol), the reference's sources
    compiled in place (oracle/_ref).  Warm-up steps are bounded (assembly, constraint and
    10 paso iterations).  Under torchrun only rank 0 works."""
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    if rank != 0:
        return
    threads = os.cpu_count() or 1
    inp = make_inputs(args.ne, args.seed, 8.0 * args.ne / 128.0)
    for _ in range(args.warmup):
        cpu_reference_warmup(inp, threads)
    vals, iters, kind = [], [], None
    t_run = time.perf_counter()
    for _ in range(args.steps):
        s = cpu_reference_solve(inp, threads, rtol=args.rtol)
        vals.append(s["time_to_solution_s"] * 1e3)
        iters.append(s["iterations"])
        kind = s["kind"]
    run_s = time.perf_counter() - t_run
    v = statistics.mean(vals)
    out = {
        "impl": "reference", "metric": METRIC, "value": round(v, 1), "unit": "ms", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(v, 1), "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic, seeded: kappa=exp(GRF corr 8 cells, std 1), 4 Gaussian blobs",
        "config": {"workload": f"Brick {args.ne}^3 variable-coefficient Poisson, u=0 on top face, "
                               f"PCG+Jacobi rtol {args.rtol:g} (assemble+constrain+solve per step)",
                   "ne": [args.ne] * 3, "seed": args.seed, "iterations": iters[0],
                   "step_ms": {"min": round(min(vals), 1), "max": round(max(vals), 1)},
                   "timed_steps_wall_s": round(run_s, 2)},
        "cpu_baseline": {"value": round(v, 1), "unit": "ms", "cores": threads, "kind": kind,
                         "sample": ("every step one complete time-to-solution on the full input: the reference's "
                                    "DefaultAssembler3D (A on the Gauss points) + insertConstraint + paso "
                                    f"Solver/PCG to rtol {args.rtol:g}; warm-up steps: assembly, constraint "
                                    "and 10 iterations")},
        "e2e": {"value": round(v, 1), "unit": "ms", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(out), flush=True)


def main():
    ap = argparse.ArgumentParser(description=__doc__.split("\n")[0])
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--ne", type=int, default=128, help="elements per axis (128 = the named workload)")
    ap.add_argument("--seed", type=int, default=2026)
    ap.add_argument("--rtol", type=float, default=RTOL,
                    help="relative residual tolerance (1e-8 = the named workload; the 256^3 "
                         "mixed-precision configuration uses 1e-10)")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline sample")
    ap.add_argument("--path", choices=["learned", "fp32"], default="learned",
                    help="timed path: learned warm start + FP32 refinement, or FP32 refinement alone")
    ap.add_argument("--sweeps", type=int, default=8, help="Chebyshev smoothing steps on the learned guess")
    ap.add_argument("--inner-tol", type=float, default=0.0,
                    help="FP32 segment reduction factor of the refinement (0: the library's default)")
    ap.add_argument("--no-batched", dest="batched", action="store_false",
                    help="skip the batched 64-system workload")
    ap.add_argument("--spmv-config", type=int, choices=[-1, 0, 1], default=-1,
                    help="FP32 iteration pipeline: -1 tuned (default); band copy 0 = 3 stages x 1 CTA/SM, "
                         "1 = 2 stages x 2 CTAs/SM; element coefficients 0 = 3 stages x 2 CTAs/SM, "
                         "1 = 2 stages x 2 CTAs/SM")
    ap.add_argument("--inner", choices=["coef", "band"], default="coef",
                    help="operator of the FP32 iterations of --path fp32 (--only fast profiling "
                         "runs): element coefficients (the timed path) or the FP32 band copy")
    ap.add_argument("--only", choices=["all", "fast", "plain", "plain_band"], default="all",
                    help="profiling runs: only the fast path, or only the plain FP64 paso solve "
                         "(CSR, or the FP64 band copy)")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
