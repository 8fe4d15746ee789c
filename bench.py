"""Benchmark: time to 1e-8 relative L2 error of the steady RT solve on one GB300.

Workload (default, --workload cfg5): the large two-strong-scatterer problem --
domain [0,2]^2, discs of radius 0.2 at (0.6, 0.6) and (1.4, 1.4) with
sigma_s = 50, sigma_t = 50.1, background sigma_t = 0.1, sigma_s = 0.01,
HG g = 0.95, beam inflow on y = 0; hp mesh from seeded refinement at the disc
edges (seed 0: 16x16 columns of 5x5 nodes and 32 angular cells of 5 nodes to
start, four rounds, up to 9 nodes per dimension), 7.95e6 DOF.  Synthetic and
seeded; no dataset.

A step is one solve from a zero initial guess to the error target.  The
reference solution is a tight plain FP64 GPU solve computed before timing
(its agreement with the CPU oracle is tested on the same recipe at 6.7e4 DOF);
the error is the quadrature-weighted relative L2 norm (weights = mass weights
with kappa = 1).  Each method's residual tolerance is calibrated (untimed) as
the loosest power of ten that reaches the 1e-8 target.  Three methods:
  plain    FP64 GMRES, sweep preconditioner (the reference-matching method)
  mixed    FP32 GMRES inside FP64 iterative refinement, sweep preconditioner
  learned  as mixed, flexible GMRES with the sweep plus the learned correction
           (network rtg/nets/sweep_correction.npz, trained by rtg.train)

value   : seconds per learned+mixed solve, device-resident inputs.
e2e     : the same solve through the C ABI with host buffers: H2D of the
          sampled forcing and inflow node values, weighting kernel, solve, D2H
          of u.  e2e_with_setup adds the handle's set-up (mesh flattening,
          coefficient sampling, tables, block inverses, autotuners, network).
roofline: the kernel that dominates the learned+mixed solve (the FP32 sweep);
          apply_roofline: the FP32 system apply, with and without the angular
          scattering matrices it streams.
adaptive_2e5: the single adaptive problem (2.2e5 DOF) with the same three
          methods, each error also stated against the CPU oracle's solution.

--workload cfg2 makes the adaptive problem the headline; --workload cfg3: 256
independent instances in one batched solve vs the same instances solved one
by one.
"""
import argparse
import ctypes as C
import json
import os
import statistics
import subprocess
import sys
import threading
import time

REPO = os.path.dirname(os.path.abspath(__file__))
for _p in (REPO, os.path.join(REPO, "radiative-transfer-amr_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import numpy as np

METRIC = "time to 1e-8 rel. L2 err: learned+mixed vs plain FP64 GPU; apply GB/s % peak"
ERR_TARGET = 1e-8


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="cfg5", choices=["cfg1", "cfg2", "cfg3", "cfg5"])
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--profile", action="store_true",
                    help="short run for ncu: each solve method, apply and sweep once in an NVTX range")
    ap.add_argument("--scale", type=float, default=1.0, help="profile mode: two-scatterer recipe scale")
    ap.add_argument("--rtol", type=float, default=1e-9, help="profile mode: solver tolerance")
    ap.add_argument("--max-it", type=int, default=3000, help="profile mode: iteration cap")
    ap.add_argument("--fp32-shape", default=None,
                    help="profile mode: pin the FP32 apply plan, 'rows,gcap,split,tc' (rtg_apply_shape)")
    return ap.parse_args()


def run_profile(args):
    """Launch sequence for ncu: set-up and one warm-up of each piece, then each
    piece once inside an NVTX range named after it -- solve_learned,
    solve_mixed, solve_plain (one solve to --rtol each), apply_fp32,
    sweep_fp32, apply_fp64, sweep_fp64 -- so that ncu --nvtx --nvtx-include
    "<name>/" captures exactly one piece.  --scale < 1 takes the two-scatterer
    recipe with fewer refinement rounds (a smaller case of the same kernels);
    --fp32-shape pins the FP32 apply plan (e.g. the tensor-core plan, which
    the autotuner picks at full size only)."""
    import torch
    from rtg import Problem, _lib, learned as LN, workloads as W
    torch.cuda.set_device(0)
    if args.workload == "cfg5" and args.scale < 1.0:
        mesh, spec = W.config5_mesh(scale=args.scale), W.two_disc_problem()
    else:
        _, mesh, spec = workload(args.workload)
    prob = Problem(spec.kappa, spec.sigma, spec.Phi, spec.f, spec.bcs_dirac)
    ctx = prob.context(mesh)
    if args.fp32_shape:
        shape = np.asarray([int(v) for v in args.fp32_shape.split(",")], dtype=np.int32)
        _lib.check(ctx.lib.rtg_apply_shape(ctx.h, _lib.RTG_FP32, _lib.ptr(shape, C.c_int32)))
    LN.set_params(ctx, LN.load(LN.DEFAULT_NET)[0])
    f_dev = ctx.forcing(spec.f)
    g_dev = ctx.inflow(spec.bcs_dirac)
    fl = _lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS
    x32 = torch.randn(ctx.N, dtype=torch.float32, device=ctx.device)
    y32 = torch.empty_like(x32)
    x64 = torch.randn(ctx.N, dtype=torch.float64, device=ctx.device)
    y64 = torch.empty_like(x64)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=ctx.device)
    pieces = [("solve_learned", lambda: ctx.solve(f_dev, g_dev, method=1, precond=3, rtol=args.rtol,
                                                  max_it=args.max_it, restart=ARMS["learned_mixed"][2],
                                                  inner_rtol=1e-5)),
              ("solve_mixed", lambda: ctx.solve(f_dev, g_dev, method=1, precond=1, rtol=args.rtol,
                                                max_it=args.max_it, restart=ARMS["mixed"][2], inner_rtol=1e-5)),
              ("solve_plain", lambda: ctx.solve(f_dev, g_dev, method=0, precond=1, rtol=args.rtol,
                                                max_it=args.max_it, restart=ARMS["plain_fp64"][2])),
              ("apply_fp32", lambda: ctx.apply(fl, x32, y32, prec=_lib.RTG_FP32)),
              ("sweep_fp32", lambda: ctx.precondition(x32, y32, prec=_lib.RTG_FP32)),
              ("apply_fp64", lambda: ctx.apply(fl, x64, y64, prec=_lib.RTG_FP64)),
              ("sweep_fp64", lambda: ctx.precondition(x64, y64, prec=_lib.RTG_FP64))]
    out = {"ndof": ctx.N, "info": ctx.info}
    for name, fn in pieces:
        fn()
    out["sweep_bytes_fp32"] = sweep_bytes(ctx, 4)[0]
    out["sweep_bytes_fp64"] = sweep_bytes(ctx, 8)[0]
    out["w_bytes_fp32"] = w_bytes_fp32(ctx)
    torch.cuda.synchronize()
    for name, fn in pieces:
        flush.fill_(1.0)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        torch.cuda.nvtx.range_push(name)
        r = fn()
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_pop()
        out[name + "_s"] = time.perf_counter() - t0
        if name.startswith("solve"):
            out[name + "_iterations"] = r[1]["iterations"]
    print(json.dumps(out))


def workload(name, seed=0):
    from rtg import workloads as W
    if name == "cfg1":
        return ("manufactured 4x4x4 cells n=4 (4096 DOF)", W.config1_mesh(), W.manufactured_problem())
    if name == "cfg5":
        return ("two strong scatterers on [0,2]^2 (sigma_s 50, sigma_t 50.1, HG g 0.95), disc-edge hp "
                "refinement seed %d: 16x16 columns x 32 angular cells to start, 5..9 nodes/dim (~7.9e6 DOF)"
                % seed, W.config5_mesh(seed=seed), W.two_disc_problem())
    return ("gaussian-bump adaptive hp, seed %d (~2.2e5 DOF)" % seed, W.config2_mesh(seed=seed),
            W.gaussian_bump_problem())


def peaks():
    try:
        with open(os.path.join(REPO, "MEASURED_PEAKS.json")) as fh:
            p = json.load(fh)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clock/throttle samples during the timed region."""

    def __init__(self, index=0):
        self.samples = []
        self.proc = None
        self.index = index

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), "--query-gpu=" + q,
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.samples.append([x.strip() for x in line.split(",")])

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for s in self.samples:
            try:
                sm.append(float(s[1]))
                mx = float(s[2])
                for k, nm in enumerate(names):
                    if s[5 + k].lower().startswith("active"):
                        reasons.add(nm)
            except Exception:
                pass
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


def rel_l2(u, ref, w):
    return float(np.sqrt(np.sum(w * (u - ref) ** 2) / np.sum(w * ref ** 2)))


def oracle_solve(mesh, spec, rtol, u_ref=None, w=None, o=None):
    """The oracle port of the path on the host (one thread): assemble the
    reference's split system with scipy (rt/solve.py:81-101) and solve it with
    scipy GMRES(50) preconditioned by the oracle's upwind sweep (this build's
    preconditioner restated on the CPU; the reference itself hands PETSc
    bjacobi or kaczmarz), to relative residual rtol.  Returns timings, the
    solution and its error against u_ref."""
    from oracle import rt_oracle as O
    t0 = time.perf_counter()
    if o is None:
        o = O.assemble(mesh, spec.kappa, spec.sigma, spec.Phi, spec.f, spec.bcs_dirac)
    t_asm = time.perf_counter() - t0
    t1 = time.perf_counter()
    u, its, info = O.solve_sweep_gmres(o, o["layout"], rtol=rtol, maxiter=400)
    t_solve = time.perf_counter() - t1
    err = rel_l2(u, u_ref, w) if u_ref is not None else None
    return {"assembly_s": t_asm, "solve_s": t_solve, "iterations": its, "rtol": rtol, "rel_l2_err": err,
            "u": u, "o": o}


def calibrated_cpu_rtol(mesh, spec, o, u_tight, w):
    """The loosest power of ten (1e-7 .. 1e-13) at which the oracle's solve
    reaches the error target against its own tight solve (untimed), the same
    rule the GPU methods use (which start at 1e-6; on these problems 1e-6
    never reaches 1e-8, and each oracle solve costs seconds)."""
    for k in range(7, 14):
        r = oracle_solve(mesh, spec, 10.0 ** (-k), u_tight, w, o=o)
        if r["rel_l2_err"] <= ERR_TARGET:
            return 10.0 ** (-k)
    return 1e-13


def cpu_baseline(mesh, spec, rtol, u_ref=None, w=None, scale=1.0, sample_desc="whole workload"):
    """Timed oracle solve (assembly + sweep-GMRES) scaled by `scale` to the
    full workload."""
    r = oracle_solve(mesh, spec, rtol, u_ref, w)
    t = r["assembly_s"] + r["solve_s"]
    return {"value": t * scale, "unit": "s", "cores": 1, "kind": "port",
            "solver": "oracle port: scipy GMRES(50) with this build's upwind sweep restated on the CPU "
                      "(not the reference's PETSc bjacobi/kaczmarz, which cannot run here)",
            "sample": "{}: oracle assembly {:.1f} s + sweep-preconditioned GMRES(50) {:.1f} s ({} iterations, "
                      "rtol {:g} calibrated to the 1e-8 error target), scaled by {:.1f}".format(
                          sample_desc, r["assembly_s"], r["solve_s"], r["iterations"], rtol, scale),
            "rel_l2_err": r["rel_l2_err"]}


def cpu_sample_cfg5(n_full):
    """Bounded sample of the two-scatterer workload for the CPU arms: the
    same recipe at 6.7e4 DOF (8x8 columns of 2x2 nodes, the same 32 angular
    cells of 5 nodes, one disc-edge refinement round), oracle solve at the
    rtol calibrated on the sample, wall time scaled by the DOF ratio (the
    per-DOF work of assembly and of one iteration is set by the angular mesh,
    which the sample shares)."""
    from oracle import rt_oracle as O
    from rtg import workloads as W
    mesh, spec = W.config5_small_mesh(rounds=1), W.two_disc_problem()
    o = O.assemble(mesh, spec.kappa, spec.sigma, spec.Phi, spec.f, spec.bcs_dirac)
    w = O.l2_weights(mesh, o["layout"])
    tight = oracle_solve(mesh, spec, 1e-13, o=o)["u"]
    rtol = calibrated_cpu_rtol(mesh, spec, o, tight, w)
    return mesh, spec, rtol, tight, w, n_full / o["N"], o["N"]


def _batch_instance_cpu(job):
    """One instance of the batched workload through the oracle port (worker of
    cpu_baseline_batch): rebuilt from its seed, assembled, solved with the
    sweep-preconditioned GMRES(50) to rtol."""
    seed, rtol = job
    from rtg import workloads as W
    from oracle import rt_oracle as O
    mesh, spec = W.batch_instance(seed)
    o = O.assemble(mesh, spec.kappa, spec.sigma, spec.Phi, spec.f, spec.bcs_dirac)
    _, its, info = O.solve_sweep_gmres(o, o["layout"], rtol=rtol)
    return its, info


def cpu_baseline_batch(seeds, rtol, n_total, workers=None):
    """The batched workload's CPU baseline on all host cores: a bounded sample
    of its instances (seeds) through the oracle port in a spawn process pool,
    wall time scaled to n_total instances."""
    import multiprocessing as mp
    workers = workers or max(1, min(len(seeds), os.cpu_count() or 1))
    t0 = time.perf_counter()
    with mp.get_context("spawn").Pool(workers) as pool:
        res = pool.map(_batch_instance_cpu, [(s, rtol) for s in seeds])
    wall = time.perf_counter() - t0
    return {"value": wall * n_total / len(seeds), "unit": "s", "cores": workers, "kind": "port",
            "sample": "{} of {} instances (seeds {}..{}), oracle assembly + scipy sweep-preconditioned GMRES(50) "
                      "to rtol {:g} in a {}-process pool, wall {:.1f} s (pool start-up included) scaled by {:.0f}"
                      .format(len(seeds), n_total, seeds[0], seeds[-1], rtol, workers, wall, n_total / len(seeds)),
            "iterations_max": max(r[0] for r in res), "all_converged": all(r[1] == 0 for r in res)}


def _events(stream):
    import torch
    return torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)


def kernel_time(fn, stream, flush, reps=20):
    """Median CUDA-event duration of fn() on the stream, L2 flushed before each."""
    import torch
    for _ in range(3):
        fn()
    durs = []
    for _ in range(reps):
        flush.fill_(1.0)
        e0, e1 = _events(stream)
        e0.record(stream)
        fn()
        e1.record(stream)
        torch.cuda.synchronize()
        durs.append(e0.elapsed_time(e1) / 1e3)
    return statistics.median(durs)


def amr_indicators(ctx, mesh, u_host, stream, flush, with_cpu):
    """The AMR step after the solve on the solution: the librtg indicator
    kernels (CUDA events, L2 flushed), the whole rtg.ErrorIndicator methods
    (host flags included, wall clock), and the CPU restatement's time (oracle
    port, one core) on the same mesh and vector."""
    import torch
    from rtg import ErrorIndicator, Projection, _lib
    N = ctx.N
    lay = ctx.layout
    ud = ctx.to_device(u_host)
    ce = torch.empty(lay.nelem, dtype=torch.float64, device=ctx.device)
    cc = torch.empty(lay.ncols, dtype=torch.float64, device=ctx.device)
    cl = torch.empty(lay.ncols, dtype=torch.float64, device=ctx.device)
    el = torch.empty(lay.nelem, dtype=torch.float64, device=ctx.device)
    lib, h, sp = ctx.lib, ctx.h, C.c_void_p(stream.cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr())
    t0 = time.perf_counter()
    _lib.check(lib.rtg_error_spatial_jump(h, p(ud), p(cc), sp))   # first call builds the pair tables
    torch.cuda.synchronize()
    setup = time.perf_counter() - t0
    t_ang = kernel_time(lambda: _lib.check(lib.rtg_error_angular_jump(h, p(ud), p(ce), p(cc), sp)), stream, flush)
    t_spt = kernel_time(lambda: _lib.check(lib.rtg_error_spatial_jump(h, p(ud), p(cc), sp)), stream, flush)
    t_hp = kernel_time(lambda: _lib.check(lib.rtg_hp_steer(h, p(ud), p(cl), p(el), sp)), stream, flush)
    proj = Projection(mesh)
    proj.from_vector(u_host)
    walls = {}
    for kind in ("angular", "spatial"):
        ts = []
        for _ in range(4):
            ind = ErrorIndicator(proj, "all", "hp", (0.5, 0.5), ctx=ctx)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            (ind.error_angular_jump if kind == "angular" else ind.error_spatial_jump)()
            ts.append(time.perf_counter() - t0)
        walls[kind] = statistics.median(ts[1:])
    out = {"workload": "indicators on the solution of the same problem", "ndof": N,
           "setup_s": setup,
           "angular_jump_us": 1e6 * t_ang, "spatial_jump_us": 1e6 * t_spt, "hp_steer_us": 1e6 * t_hp,
           "error_angular_jump_method_s": walls["angular"], "error_spatial_jump_method_s": walls["spatial"],
           "dof_per_s_spatial_jump": N / t_spt}
    if with_cpu:
        from oracle import amr_oracle as AO
        t0 = time.perf_counter()
        AO.indicator(mesh, u_host, "ang", "all", "hp", (0.5, 0.5))
        t1 = time.perf_counter()
        AO.indicator(mesh, u_host, "spt", "all", "hp", (0.5, 0.5))
        t2 = time.perf_counter()
        out["cpu_baseline"] = {"kind": "port", "cores": 1, "angular_s": t1 - t0, "spatial_s": t2 - t1,
                               "sample": "whole mesh: oracle restatement (numpy) of error_angular_jump and "
                                         "error_spatial_jump with the flags and hp steering they trigger"}
    return out


def profiled_traffic(name):
    """DRAM bytes per launch recorded from an ncu capture in profiles/<name>.md
    (line "traffic_bytes_per_launch: N"), or None."""
    try:
        with open(os.path.join(REPO, "profiles", name + ".md")) as fh:
            for line in fh:
                if line.startswith("traffic_bytes_per_launch:"):
                    return int(line.split(":", 1)[1])
    except OSError:
        pass
    return None


def sweep_bytes(ctx, prec_bytes):
    """Algorithmic bytes of one sweep kernel: read r, write z, read the element
    block inverses and the upwind maps of the one-phase elements (both BF16 for
    the FP32 sweep, FP64 for the FP64 one) and the maps' upwind value indices
    (8 bytes each); upwind face values re-read through L2 count 0."""
    from rtg import _lib
    lev, lag, inv = C.c_int(), C.c_int(), C.c_int64()
    _lib.check(ctx.lib.rtg_sweep_info(ctx.h, C.byref(lev), C.byref(lag), C.byref(inv), None))
    one, gm, up = C.c_int(), C.c_int64(), C.c_int64()
    prec = _lib.RTG_FP32 if prec_bytes == 4 else _lib.RTG_FP64
    _lib.check(ctx.lib.rtg_sweep_maps(ctx.h, prec, C.byref(one), C.byref(gm), C.byref(up), None))
    blk_bytes = 2 if prec_bytes == 4 else 8
    total = 2 * prec_bytes * ctx.N + blk_bytes * (inv.value + gm.value) + 8 * up.value
    return int(total), int(lev.value), int(lag.value)


def l2_weights_dev(ctx, spec):
    """Quadrature weights (dx dy dth / 8) wx wy wth (mass weights with kappa = 1)."""
    import torch
    from rtg import _lib
    X, Y, _ = ctx.layout.node_coords()
    ones = ctx.apply(_lib.RTG_MASS, torch.ones(ctx.N, dtype=torch.float64, device=ctx.device))
    kap = ctx.to_device(np.asarray(np.broadcast_to(spec.kappa(X, Y), (ctx.N,)), dtype=np.float64))
    return (ones / kap).cpu().numpy()


def setup_context(mesh, spec, params):
    """Handle creation and every first-use set-up, timed: mesh flattening and
    coefficient sampling with the table upload, forcing and inflow vectors,
    the sweep's block inverses in both precisions, the apply autotuners in
    both precisions, the network's coefficients."""
    import torch
    from rtg import Problem, _lib, learned as LN
    out = {}
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    prob = Problem(spec.kappa, spec.sigma, spec.Phi, spec.f, spec.bcs_dirac)
    ctx = prob.context(mesh)
    torch.cuda.synchronize()
    out["context_s"] = time.perf_counter() - t0
    t0 = time.perf_counter()
    f_dev = ctx.forcing(spec.f)
    g_dev = ctx.inflow(spec.bcs_dirac)
    torch.cuda.synchronize()
    out["vectors_s"] = time.perf_counter() - t0
    # inputs and outputs of both precisions made before the clocks start: the
    # timed regions hold the library's own first-use work only
    z64 = torch.zeros(ctx.N, dtype=torch.float64, device=ctx.device)
    z32 = torch.zeros(ctx.N, dtype=torch.float32, device=ctx.device)
    o64, o32 = torch.empty_like(z64), torch.empty_like(z32)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    ctx.precondition(z64, o64)
    ctx.precondition(z32, o32, prec=_lib.RTG_FP32)
    torch.cuda.synchronize()
    out["sweep_setup_s"] = time.perf_counter() - t0
    t0 = time.perf_counter()
    ctx.apply(_lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS, z64, o64)
    ctx.apply(_lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS, z32, o32, prec=_lib.RTG_FP32)
    torch.cuda.synchronize()
    out["apply_tuning_s"] = time.perf_counter() - t0
    t0 = time.perf_counter()
    LN.set_params(ctx, params)
    torch.cuda.synchronize()
    out["network_s"] = time.perf_counter() - t0
    out["total_s"] = sum(out.values())
    return ctx, f_dev, g_dev, out


# (method, preconditioner, GMRES restart length): each method's restart is
# the fastest of 10, 15, 20, 25, 30, 40, 50 on the two-scatterer problem
# (plain FP64: 30; the FP32 inner solves of the mixed methods: 15, where a
# shorter basis saves Gram-Schmidt work without adding iterations)
ARMS = {"plain_fp64": (0, 1, 30), "mixed": (1, 1, 15), "learned_mixed": (1, 3, 15)}


def solve_arm(ctx, f_dev, g_dev, arm, rtol):
    method, pc, restart = ARMS[arm]
    return ctx.solve(f_dev, g_dev, method=method, rtol=rtol, max_it=3000, precond=pc, restart=restart,
                     inner_rtol=1e-5)


def measure_arms(ctx, f_dev, g_dev, u_ref_h, w, steps, warmup, flush, stream, clk=None, u_oracle=None):
    """Calibrate each method's rtol against the reference solution, then time
    it (learned+mixed: steps after warmup; the others: up to 3 after 1)."""
    import torch
    rtols, first = {}, {}
    for arm in ARMS:
        for k in range(6, 15):
            t0 = time.perf_counter()
            u, info = solve_arm(ctx, f_dev, g_dev, arm, 10.0 ** (-k))
            torch.cuda.synchronize()
            first.setdefault(arm, time.perf_counter() - t0)
            if rel_l2(u.cpu().numpy(), u_ref_h, w) <= ERR_TARGET:
                rtols[arm] = 10.0 ** (-k)
                break
        else:
            raise RuntimeError("{} did not reach the error target".format(arm))
    launch_count = ctx.lib.rtg_launch_count
    res = {}
    for arm in ("learned_mixed", "mixed", "plain_fp64"):
        n_steps, n_warm = (steps, warmup) if arm == "learned_mixed" else (max(1, min(steps, 3)), 1)
        for _ in range(n_warm):
            solve_arm(ctx, f_dev, g_dev, arm, rtols[arm])
        times, errs, infos, launched = [], [], [], 0
        if clk is not None and arm == "learned_mixed":
            clk.__enter__()
        for _ in range(n_steps):
            flush.fill_(1.0)
            torch.cuda.synchronize()
            e0, e1 = _events(stream)
            n0 = launch_count()
            e0.record(stream)
            u, info = solve_arm(ctx, f_dev, g_dev, arm, rtols[arm])
            e1.record(stream)
            launched += launch_count() - n0
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1) / 1e3)
            uh = u.cpu().numpy()
            errs.append(rel_l2(uh, u_ref_h, w))
            infos.append(info)
        if clk is not None and arm == "learned_mixed":
            clk.__exit__()
        i = infos[-1]
        res[arm] = {"rtol": rtols[arm], "restart": ARMS[arm][2], "rel_l2_err": max(errs),
                    "median_s": statistics.median(times),
                    "seconds": times, "iterations": i["iterations"], "outer": i["outer"],
                    "fp64_applies": i["fp64_applies"], "fp32_applies": i["fp32_applies"],
                    "learned": i["learned"], "fallbacks": i["fallbacks"], "first_solve_s": first[arm],
                    "learned_kept": i["learned_kept"],
                    "launches_per_solve": launched // max(1, n_steps)}
        if u_oracle is not None:
            res[arm]["rel_l2_err_vs_oracle"] = rel_l2(uh, u_oracle, w)
    return res


def w_bytes_fp32(ctx):
    """Bytes of the FP32 angular scattering matrices an FP32 apply streams
    (one Nth_col x Nth_col matrix per distinct column angular mesh)."""
    so = ctx.sampled.sig_off
    return int(4 * (so[-1] - so[0]))


def run_ours(args):
    if args.workload == "cfg3":
        return run_batched(args)
    import torch
    from rtg import _lib, learned as LN

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", init_method="env://")
        torch.cuda.set_device(local)
    else:
        torch.cuda.set_device(0)
    t0 = time.perf_counter()
    desc, mesh, spec = workload(args.workload, seed=rank)
    mesh_s = time.perf_counter() - t0
    params, net_meta = LN.load(LN.DEFAULT_NET)
    ctx, f_dev, g_dev, setup = setup_context(mesh, spec, params)
    N = ctx.N
    w = l2_weights_dev(ctx, spec)
    # reference solution: tight plain FP64 solve
    u_ref, info_ref = ctx.solve(f_dev, g_dev, method=0, rtol=1e-13, max_it=3000, precond=1)
    u_ref_h = u_ref.cpu().numpy()
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=ctx.device)
    stream = torch.cuda.current_stream()
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    clk = ClockSampler(torch.cuda.current_device())
    res = measure_arms(ctx, f_dev, g_dev, u_ref_h, w, args.steps, args.warmup, flush, stream, clk=clk)
    if world > 1:
        torch.distributed.barrier()

    # e2e through the C ABI with host buffers (learned+mixed)
    lib = ctx.lib
    fvals = torch.from_numpy(ctx.node_values(spec.f)).pin_memory()
    gvals = torch.from_numpy(np.ascontiguousarray(g_dev.cpu().numpy())).pin_memory()
    u_host = torch.empty(N, dtype=torch.float64).pin_memory()
    fd = torch.empty(N, dtype=torch.float64, device=ctx.device)
    fw = torch.empty_like(fd)
    gd = torch.empty_like(fd)
    ud = torch.zeros_like(fd)
    opts = _lib.SolveOpts(method=1, restart=ARMS["learned_mixed"][2], max_it=3000, rtol=res["learned_mixed"]["rtol"],
                          atol=0.,
                          precond=3, nonzero_guess=0, inner_rtol=1e-5, max_outer=20, verbose=0)
    sinfo = _lib.SolveInfo()
    sp = C.c_void_p(stream.cuda_stream)
    e2e_times = []
    for it in range(args.warmup + args.steps):
        flush.fill_(1.0)
        torch.cuda.synchronize()
        e0, e1 = _events(stream)
        e0.record(stream)
        fd.copy_(fvals, non_blocking=True)
        gd.copy_(gvals, non_blocking=True)
        _lib.check(lib.rtg_weight_forcing(ctx.h, C.c_void_p(fd.data_ptr()), C.c_void_p(fw.data_ptr()), sp))
        _lib.check(lib.rtg_solve(ctx.h, C.c_void_p(fw.data_ptr()), C.c_void_p(gd.data_ptr()),
                                 C.c_void_p(ud.data_ptr()), C.byref(opts), C.byref(sinfo), None, 0, sp))
        u_host.copy_(ud, non_blocking=True)
        e1.record(stream)
        torch.cuda.synchronize()
        if it >= args.warmup:
            e2e_times.append(e0.elapsed_time(e1) / 1e3)
    e2e_err = rel_l2(u_host.numpy(), u_ref_h, w)

    # rooflines: the FP32 sweep (dominant kernel of the learned+mixed solve) and the FP32 apply
    peak, peak_kind = peaks()
    r32 = torch.randn(N, dtype=torch.float32, device=ctx.device)
    z32 = torch.empty_like(r32)
    t_sweep = kernel_time(lambda: ctx.precondition(r32, z32, prec=_lib.RTG_FP32), stream, flush)
    sb, nlev, nlag = sweep_bytes(ctx, 4)
    t_apply = kernel_time(lambda: ctx.apply(_lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS, r32, z32, prec=_lib.RTG_FP32),
                          stream, flush)
    bytes_apply = int(ctx.info["bytes_per_apply_fp32"])
    wb = w_bytes_fp32(ctx)
    x64 = torch.randn(N, dtype=torch.float64, device=ctx.device)
    y64 = torch.empty_like(x64)
    t_apply64 = kernel_time(lambda: ctx.apply(_lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS, x64, y64, prec=_lib.RTG_FP64),
                            stream, flush, 5)
    t_sweep64 = kernel_time(lambda: ctx.precondition(x64, y64, prec=_lib.RTG_FP64), stream, flush, 5)

    t_l = res["learned_mixed"]["seconds"]
    value = statistics.median(t_l)
    if world > 1:
        tt = torch.tensor([max(t_l)], device=ctx.device)
        torch.distributed.all_reduce(tt, op=torch.distributed.ReduceOp.MAX)
        value = float(tt.item())
    if rank != 0:
        return None
    t_plain = res["plain_fp64"]["median_s"]
    tag = "cfg5" if args.workload == "cfg5" else "cfg2"
    e2e = statistics.median(e2e_times)
    sweep_traffic = profiled_traffic("sweep_persistent_kernel_fp32_" + tag)
    apply_traffic = profiled_traffic("apply_tiled_kernel_fp32_" + tag)
    out = {
        "metric": METRIC, "value": value, "unit": "s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1e3 * value, "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32-inner/f64-outer",
        "data": "synthetic (seeded hp mesh and coefficients)",
        "config": {"workload": desc, "ndof": N, "ndof_interior": int(ctx.info["ndof_interior"]),
                   "error_target": ERR_TARGET, "l2_flush": "256 MB write before every timed solve and kernel",
                   "learned_mixed": res["learned_mixed"], "mixed": res["mixed"], "plain_fp64": res["plain_fp64"],
                   "speedup_learned_mixed_vs_plain_fp64": t_plain / value,
                   "speedup_mixed_vs_plain_fp64": t_plain / res["mixed"]["median_s"],
                   "network": {"file": "rtg/nets/sweep_correction.npz", **net_meta},
                   "reference_solution": {"method": "plain FP64 GPU solve", "rtol": 1e-13,
                                          "iterations": info_ref["iterations"],
                                          "rel_residual": info_ref["res_f"] / max(info_ref["rhs_norm"], 1e-300)},
                   "setup": {"mesh_s": mesh_s, **setup},
                   "kernels_us": {"sweep_fp32": 1e6 * t_sweep, "sweep_fp64": 1e6 * t_sweep64,
                                  "apply_fp32": 1e6 * t_apply, "apply_fp64": 1e6 * t_apply64},
                   "apply_fp64": {"flops": int(ctx.info["flops_per_apply"]),
                                  "note": "tiled kernel FP64-pipe bound (GB300 FP64 rate is 1/64 of FP32), the product on the tensor cores in digits"},
                   "sweep": {"levels": nlev, "lagged_couplings": nlag},
                   "parallelism": "replicas" if world > 1 else "single GPU"},
        "e2e": {"value": e2e, "unit": "s", "h2d_bytes_per_step": 2 * 8 * N,
                "d2h_bytes_per_step": 8 * N, "rel_l2_err": e2e_err},
        "e2e_with_setup": {"value": e2e + setup["total_s"] + mesh_s, "unit": "s",
                           "note": "e2e plus the handle's set-up (a new mesh in an AMR loop pays it per solve)"},
        "gpu_launches": int(res["learned_mixed"]["launches_per_solve"]) * args.steps,
        "roofline": {"bound": "hbm", "achieved": sb / t_sweep / 1e9, "peak": peak, "unit": "GB/s",
                     "frac": sb / t_sweep / 1e9 / peak, "traffic": sweep_traffic,
                     "frac_of_traffic": (sweep_traffic / t_sweep / 1e9 / peak) if sweep_traffic else None,
                     "kernel": "sweep_persistent_kernel<float>", "bytes_per_launch": sb, "launch_s": t_sweep,
                     "peak_kind": peak_kind,
                     "note": "bytes_per_launch counts every element's reads of its block inverse and of the "
                             "map it uses (one-phase elements); elements with identical blocks share them, so the "
                             "DRAM traffic (ncu) is lower and part of the bytes come from L2; {} wavefront levels, "
                             "{:.2f} us per level".format(
                                 nlev, 1e6 * t_sweep / max(nlev, 1))},
        "apply_roofline": {"bound": "hbm", "achieved": bytes_apply / t_apply / 1e9, "peak": peak, "unit": "GB/s",
                           "frac": bytes_apply / t_apply / 1e9 / peak, "kernel": "apply_tiled_kernel (FP32 system)",
                           "bytes_per_launch": bytes_apply, "w_bytes_per_launch": wb,
                           "frac_with_w": (bytes_apply + wb) / t_apply / 1e9 / peak,
                           "traffic": apply_traffic,
                           "frac_of_traffic": (apply_traffic / t_apply / 1e9 / peak) if apply_traffic else None,
                           "launch_s": t_apply, "peak_kind": peak_kind, "dof_applies_per_s": N / t_apply,
                           "tflops": ctx.info["flops_per_apply"] / t_apply / 1e12},
        "clocks": clk.summary(),
    }
    if args.workload == "cfg5":
        if not args.no_cpu:
            smesh, sspec, srtol, stight, sw, scale, sN = cpu_sample_cfg5(N)
            out["cpu_baseline"] = cpu_baseline(smesh, sspec, srtol, stight, sw, scale=scale,
                                               sample_desc="the same recipe at {} DOF (one refinement round, "
                                                           "8x8 columns of 2x2 nodes)".format(sN))
        out["adaptive_2e5"] = secondary_adaptive(args, flush, stream)
        out["batched_256"] = batched_measure(2, 1, not args.no_cpu, cpu_instances=16)
    else:
        out["amr_indicators"] = amr_indicators(ctx, mesh, u_ref_h, stream, flush, not args.no_cpu)
        if not args.no_cpu:
            out["cpu_baseline"] = cpu_baseline(mesh, spec, res["plain_fp64"]["rtol"], u_ref_h, w)
    ctx.close()
    return out


def secondary_adaptive(args, flush, stream):
    """The single adaptive problem (2.2e5 DOF): the three methods timed the same
    way, each error also against the CPU oracle's solution; the AMR indicator
    kernels; the oracle's solve timed as its CPU baseline."""
    from rtg import learned as LN
    desc, mesh, spec = workload("cfg2")
    params, _ = LN.load(LN.DEFAULT_NET)
    ctx, f_dev, g_dev, setup = setup_context(mesh, spec, params)
    w = l2_weights_dev(ctx, spec)
    u_ref, _ = ctx.solve(f_dev, g_dev, method=0, rtol=1e-14, max_it=3000, precond=1)
    u_ref_h = u_ref.cpu().numpy()
    orc = oracle_solve(mesh, spec, 1e-13, u_ref_h, w)
    res = measure_arms(ctx, f_dev, g_dev, u_ref_h, w, min(args.steps, 3), 1, flush, stream, u_oracle=orc["u"])
    out = {"workload": desc, "ndof": ctx.N, "setup": setup, **res,
           "speedup_learned_mixed_vs_plain_fp64": res["plain_fp64"]["median_s"] / res["learned_mixed"]["median_s"],
           "gpu_reference_vs_oracle_rel_l2": orc["rel_l2_err"],
           "oracle_solution": {"rtol": 1e-13, "iterations": orc["iterations"]}}
    out["amr_indicators"] = amr_indicators(ctx, mesh, u_ref_h, stream, flush, not args.no_cpu)
    if not args.no_cpu:
        out["cpu_baseline"] = cpu_baseline(mesh, spec, res["plain_fp64"]["rtol"], u_ref_h, w)
    ctx.close()
    return out


def batched_measure(steps, warmup, with_cpu, cpu_instances=32):
    """cfg3: 256 independent instances (seeded degree, size, sigma_t, albedo,
    g) in one batched solve (method 1, one handle, graph-captured restart
    cycle), against solving the same instances one by one through rt.Problem-
    style contexts.  Each instance's error is measured against its own tight
    FP64 solve."""
    import torch
    from rtg import DeviceContext, _lib, workloads as W
    from rtg.batch import BatchContext
    nb = 256
    inst = [W.batch_instance(1000 + k) for k in range(nb)]
    t0 = time.perf_counter()
    bc = BatchContext(inst)
    f = bc.forcing()
    g = bc.inflow()
    torch.cuda.synchronize()
    setup_s = time.perf_counter() - t0
    stream = torch.cuda.current_stream()
    # reference solutions: tight individual FP64 solves
    ctxs = [DeviceContext(m, p.kappa, p.sigma, p.Phi) for m, p in inst]
    fs = [c.forcing(p.f) for c, (m, p) in zip(ctxs, inst)]
    gs = [c.inflow(p.bcs_dirac) for c, (m, p) in zip(ctxs, inst)]
    refs = [c.solve(fi, gi, method=0, precond=1, rtol=1e-13, max_it=20000)[0] for c, fi, gi in zip(ctxs, fs, gs)]

    def errors(parts):
        return [float(torch.linalg.norm(a - r) / torch.linalg.norm(r)) for a, r in zip(parts, refs)]

    rtol = None
    for k in range(6, 14):
        u, infos = bc.solve(f, g, rtol=10.0 ** (-k), inner_rtol=1e-5)
        if max(errors(bc.split(u))) <= ERR_TARGET:
            rtol = 10.0 ** (-k)
            break
    if rtol is None:
        raise RuntimeError("batched solve did not reach the error target")
    for _ in range(warmup):
        bc.solve(f, g, rtol=rtol, inner_rtol=1e-5)
    times = []
    launch_count = _lib.load().rtg_launch_count
    n_launch = 0
    with ClockSampler(0) as clk:
        for _ in range(steps):
            torch.cuda.synchronize()
            e0, e1 = _events(stream)
            n0 = launch_count()
            e0.record(stream)
            u, infos = bc.solve(f, g, rtol=rtol, inner_rtol=1e-5)
            e1.record(stream)
            n_launch += launch_count() - n0
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1) / 1e3)
    errs = errors(bc.split(u))
    seq = []
    for _ in range(2):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for c, fi, gi in zip(ctxs, fs, gs):
            c.solve(fi, gi, method=1, precond=1, rtol=rtol, inner_rtol=1e-5, restart=30)
        torch.cuda.synchronize()
        seq.append(time.perf_counter() - t0)
    for c in ctxs:
        c.close()
    value = statistics.median(times)
    out = {"value": value, "unit": "s", "steps": steps, "warmup": warmup, "n_instances": nb,
           "workload": "256 independent instances (batch_instance seeds 1000..1255)", "ndof": int(bc.N),
           "rtol": rtol, "max_rel_err": max(errs), "error_target": ERR_TARGET, "setup_s": setup_s,
           "sequential_one_by_one_s": min(seq), "speedup_batched_vs_sequential": min(seq) / value,
           "iterations_max": max(i["iterations"] for i in infos), "gpu_launches": int(n_launch),
           "clocks": clk.summary()}
    if with_cpu:
        # all host cores, a bounded sample of the 256 instances
        out["cpu_baseline"] = cpu_baseline_batch(list(range(1000, 1000 + cpu_instances)), rtol, nb)
    return out


def run_batched(args):
    rank = int(os.environ.get("RANK", "0"))
    import torch
    torch.cuda.set_device(0)
    b = batched_measure(args.steps, args.warmup, not args.no_cpu)
    if rank != 0:
        return None
    out = {"metric": METRIC, "value": b["value"], "unit": "s", "n_gpus": 1, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": 1e3 * b["value"], "higher_is_better": False, "scaling": "weak",
           "vs_baseline": None, "dtype": "f32-inner/f64-outer", "data": "synthetic (256 seeded instances)",
           "config": {k: b[k] for k in ("workload", "ndof", "rtol", "max_rel_err", "error_target", "setup_s",
                                        "sequential_one_by_one_s", "speedup_batched_vs_sequential",
                                        "iterations_max")},
           "e2e": {"value": b["value"], "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0,
                   "note": "inputs resident; the batched entry point takes device vectors"},
           "gpu_launches": b["gpu_launches"], "clocks": b["clocks"]}
    if "cpu_baseline" in b:
        out["cpu_baseline"] = b["cpu_baseline"]
    return out


def run_reference(args):
    """The CPU arm: the oracle port timed on the host.  Two-scatterer workload:
    each step times the bounded sample of cpu_sample_cfg5 (the rtol calibrated
    on it, untimed) and scales it to the full DOF count; the adaptive problem
    is timed whole."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return None
    desc, mesh, spec = workload(args.workload)
    if args.workload == "cfg5":
        from rtg.layout import MeshLayout
        n_full = MeshLayout(mesh).N
        smesh, sspec, rtol, tight, w, scale, sN = cpu_sample_cfg5(n_full)
        run = lambda: cpu_baseline(smesh, sspec, rtol, tight, w, scale=scale,
                                   sample_desc="the same recipe at {} DOF (one refinement round, "
                                               "8x8 columns of 2x2 nodes)".format(sN))
    else:
        from oracle import rt_oracle as O
        o = O.assemble(mesh, spec.kappa, spec.sigma, spec.Phi, spec.f, spec.bcs_dirac)
        w = O.l2_weights(mesh, o["layout"])
        tight = oracle_solve(mesh, spec, 1e-13, o=o)["u"]
        rtol = calibrated_cpu_rtol(mesh, spec, o, tight, w)
        run = lambda: cpu_baseline(mesh, spec, rtol, tight, w)
    vals = []
    for it in range(args.warmup + args.steps):
        cb = run()
        if it >= args.warmup:
            vals.append(cb["value"])
    v = statistics.median(vals)
    cb["value"] = v
    return {"metric": METRIC, "value": v, "unit": "s", "n_gpus": int(os.environ.get("WORLD_SIZE", "1")),
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * v, "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": desc}, "impl": "reference", "cpu_baseline": cb,
            "e2e": {"value": v, "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}


def main():
    args = parse()
    if args.profile:
        run_profile(args)
        return
    out = run_reference(args) if args.impl == "reference" else run_ours(args)
    if out is not None:
        print(json.dumps(out))


if __name__ == "__main__":
    main()
