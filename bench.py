#!/usr/bin/env python
"""SW2 implicit time steps per second on the 4M-triangle wet/dry beach.

Workload: 40 km x 10 km sloping beach (bed -20 m .. +3 m plus N(0, 0.2 m) noise,
seed 3), jittered Delaunay of a 2828 x 707 grid = 3 991 724 triangles, 1 999 396
nodes, 5 998 188 dofs; inflow hydrograph Q(t) = 500 + 1500 sin^2(pi t / 6 h) as a
velocity BC, dt = 120 s.  Synthetic input generated here; every array is far larger
than L2.

A "step" is one dt interval of the time loop (SW2Simulation.advance): fe_newton to the
Newton tolerance (FD Jacobian, CSR assembly, Dirichlet/scaling, preconditioned Krylov
solve per Newton iteration); a solve that fails is undone and the interval covered in
steps of dt x 0.25, as the reference's tc_scale shrinks dt.  `value` counts completed
intervals only.  A solve succeeds when max|R| <= tol_nonlin_rel * max|R(sol_old)|, or
when the increment is below inc_nonlin after a linear solve that reached its target.

Two paths are timed over the same intervals from the same state after warm-up:
  * fast:  GMRES cycles in FP32 (basis, SpMV, AMG) inside FP64 refinement and, with
           --guess learned, the message-passing network's initial guess;
  * plain: everything FP64, previous-step initial guess.
`value` is the fast path (the product); the plain path, the error between the two final
states, and both paths' error against the reference's own run on a 240 x 60 sample of
the same beach are reported beside it.

`python bench.py --impl reference` times the reference's own C code (compiled from its
sources, UMFPACK replaced by a banded LU) on the host cores for that sample and
extrapolates to the full beach (a lower bound on its CPU time).
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

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

METRIC = "SW2 timesteps/s @4M tris: learned+FP32-Krylov vs plain FP64 GPU at equal Newton tol"
UNIT = "timesteps/s"
NTRI_FULL = 3991724
SAMPLE_NX, SAMPLE_NY = 240, 60            # reference CPU sample: same beach, coarser grid


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=5)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--workload", choices=["beach4M", "basin1M", "basin1M-hydro", "estuary16M"], default="beach4M",
                   help="beach4M: the benchmark configuration; basin1M (fully wet tidal basin, dt 300 s), "
                        "basin1M-hydro (the basin under a held-out inflow hydrograph, with the basin-trained "
                        "learned guess) and estuary16M (partial wet/dry estuary, dt 180 s) measure the other "
                        "GPU configurations")
    p.add_argument("--nx", type=int, default=2828)
    p.add_argument("--ny", type=int, default=707)
    p.add_argument("--krylov-tol", type=float, default=1e-6,
                   help="inexact-Newton forcing: linear residual <= tol * Newton residual (floor: a tenth of "
                        "tol_nonlin with the relative Newton test, a hundredth with the absolute one)")
    p.add_argument("--guess", choices=["none", "learned"], default="learned")
    p.add_argument("--weights", default=None, help="trained initial-guess weights (default: the committed ones)")
    p.add_argument("--tol-rel", type=float, default=1e-8,
                   help="Newton test max|R| <= tol_rel * max|R(previous step)|; 0: the reference's absolute 1e-8")
    p.add_argument("--basis", type=int, choices=[32, 64], default=32,
                   help="fast path: FP32 (default) or FP64 GMRES basis around the FP32 preconditioner")
    p.add_argument("--restart", type=int, default=100, help="GMRES restart length of both paths (1..200)")
    p.add_argument("--no-plain", action="store_true")
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu-baseline", action="store_true")
    return p.parse_args()


# ----------------------------------------------------------------------------- helpers
class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled every 200 ms while running."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def __enter__(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.f,
                                      stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None
        return self

    def __exit__(self, *a):
        if self.p is not None:
            self.p.terminate()
            try:
                self.p.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.p.kill()

    def summary(self):
        self.f.flush()
        rows = []
        with open(self.f.name) as fh:
            for line in fh:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) >= 9:
                    rows.append(parts)
        os.unlink(self.f.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower().startswith("active")})
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": float(rows[0][2]) if rows[0][2].replace(".", "").isdigit() else None,
                "reasons": reasons, "samples": len(rows)}


def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        backend = "nccl" if args.impl == "ours" else "gloo"
        dist.init_process_group(backend, timeout=datetime.timedelta(seconds=600))
    return world, rank, local, dist


def max_over_ranks(x, dist, device="cuda"):
    """The slowest rank's value (every rank calls this at the same point)."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ----------------------------------------------------------------------------- CPU reference sample
def cpu_sample_case(nsteps):
    from adh_kraken_b200.mesh import beach_case
    return beach_case(nx=SAMPLE_NX, ny=SAMPLE_NY, nsteps=nsteps)


def start_cpu_reference(nsteps_total):
    """The reference's fe_newton (compiled from its C sources) on the SAMPLE_NX x SAMPLE_NY
    beach in a background process; its final state is kept for the error check."""
    from oracle import refio
    case = cpu_sample_case(nsteps_total)
    return case, refio.HarnessRun("run", case, extra=(nsteps_total,))


def cpu_baseline_failed(e):
    """What the bench line says of a baseline that could not be started or finished: reported, not fatal."""
    return {"value": None, "unit": UNIT, "cores": 1, "kind": "reference", "sample": f"failed: {e}"}


def begin_cpu_baseline(nsteps_total):
    """((case, run) of the reference started in the background, None), or (None, what the bench line reports)
    where it cannot be started, as without its harness."""
    try:
        return start_cpu_reference(nsteps_total), None
    except Exception as e:  # noqa: BLE001
        return None, cpu_baseline_failed(e)


def cpu_reference_result(run, case, skip):
    rec = run.wait(timeout=3600)
    secs = np.asarray(rec["step_seconds"], dtype=np.float64)
    ok = np.asarray(rec["step_ok"])
    use = secs[skip:] if len(secs) > skip else secs
    per_full = float(np.mean(use)) * NTRI_FULL / case.ntri
    sample = (f"reference fe_newton (its own C code compiled here, banded LU in place of UMFPACK, single-threaded) "
              f"on the {SAMPLE_NX}x{SAMPLE_NY} beach ({case.ntri} tris, same dt and forcing): steps {skip + 1}.."
              f"{len(secs)} at {float(np.mean(use)):.3f} s/step, {int(ok.sum())}/{len(ok)} steps converged; "
              f"extrapolated linearly by triangle count to {NTRI_FULL} tris, a lower bound on the reference's "
              f"CPU time there (its LU scales worse than linearly)")
    final = rec["sol_kept"].reshape(-1, 3 * case.nnodes)[-1] if len(rec["sol_kept"]) else None
    return 1.0 / per_full, per_full, sample, final


# ----------------------------------------------------------------------------- reference arm
def run_reference(args, world, rank, dist):
    if rank != 0:
        return
    if not os.path.exists(os.path.join(HERE, "oracle", "_ref", "adh_ref_harness")):
        print(json.dumps({"impl": "reference", "unavailable": "reference harness not built (oracle/_ref)"}))
        return
    case, run = start_cpu_reference(args.warmup + args.steps)
    value, per_full, sample, _ = cpu_reference_result(run, case, args.warmup)
    out = {"metric": METRIC, "value": value, "unit": UNIT, "impl": "reference", "n_gpus": args.gpus,
           "steps": args.steps, "warmup": args.warmup, "ms_per_step": per_full * 1e3,
           "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
           "config": {"workload": "beach4M", "ntri": NTRI_FULL, "dt_s": 120.0, "tol_nonlin": 1e-8,
                      "sample_ntri": case.ntri, "timing": "measured on the sample, extrapolated (lower bound)"},
           "cpu_baseline": {"value": value, "unit": UNIT, "cores": 1, "kind": "reference", "sample": sample},
           "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out), flush=True)


# ----------------------------------------------------------------------------- our arm
def rel_errors(a, b):
    """max |a - b| / max |b| per variable (h, u, v) of two node-major states"""
    return [float(np.abs(a[k::3] - b[k::3]).max() / max(np.abs(b[k::3]).max(), 1e-300)) for k in range(3)]


def interval_summary(recs):
    ok = [r for r in recs if r["success"]]
    out = {"intervals": len(recs), "intervals_ok": len(ok), "failed_intervals": len(recs) - len(ok),
           "dt_cuts": [r["dt_cuts"] for r in recs], "substeps": [r["substeps"] for r in recs],
           "step_start_s": [r.get("step_start") for r in recs],
           "newton_its": [r["newton_its"] for r in recs], "krylov_its": [r["krylov_its"] for r in recs],
           "final_resid": [r.get("resid_max") for r in recs], "tol_used": [r.get("tol_used") for r in recs],
           "linear_unconverged": [r.get("linear_unconverged", 0) for r in recs]}
    out["converged_by_residual"] = sum(1 for r in recs if r["success"] and r.get("resid_max") is not None
                                       and r.get("tol_used") is not None and r["resid_max"] <= r["tol_used"])
    return out


def run_ours(args, world, rank, local, dist):
    import torch
    from adh_kraken_b200.capi import default_opts, NewtonStats, lib
    from adh_kraken_b200.mesh import beach_case
    from adh_kraken_b200.timeloop import SW2Simulation, DT_REDUCE_FACTOR
    import ctypes as C

    torch.cuda.set_device(local)
    K, W = args.steps, args.warmup
    cpu_run, cpu = None, None
    if rank == 0 and world == 1 and not args.no_cpu_baseline and args.workload == "beach4M":
        cpu_run, cpu = begin_cpu_baseline(W + K)    # CPU work in the background while the GPU runs
    if args.workload == "basin1M":
        from adh_kraken_b200.mesh import basin_case
        case = basin_case(n=707, seed=2, nsteps=W + 2 * K + 8)
    elif args.workload == "basin1M-hydro":
        from adh_kraken_b200.mesh import basin_hydro_case
        case = basin_hydro_case(48, n=707, nsteps=W + 2 * K + 8)     # a hydrograph the weights never saw
    elif args.workload == "estuary16M":
        from adh_kraken_b200.mesh import estuary_case
        case = estuary_case(nsteps=W + 2 * K + 8)
    else:
        case = beach_case(nx=args.nx, ny=args.ny, nsteps=W + 2 * K + 8)
    base = dict(tol_nonlin=1e-8, tol_nonlin_rel=args.tol_rel, inc_nonlin=1e-6, max_nonlin_it=10,
                krylov_max_it=20000, krylov_tol=args.krylov_tol, precond=2, krylov_method=1,
                krylov_restart=args.restart)
    opts_fast = default_opts(krylov_precision=32, krylov_basis_precision=args.basis, **base)
    opts_plain = default_opts(krylov_precision=64, **base)
    guesser = None
    if args.guess == "learned" and args.workload in ("beach4M", "basin1M-hydro"):
        from adh_kraken_b200 import learned
        default_w = learned.WEIGHTS if args.workload == "beach4M" else learned.BASIN_WEIGHTS
        guesser = learned.load_guesser(case, args.weights or default_w)
    if guesser is not None:
        opts_fast.use_guess = 1

    def guess_hook(sim, h):
        if guesser is not None and h == case.dt:
            guesser.predict_into(sim)           # device-side guess from the resident state
        elif guesser is not None:
            sim.model.set_guess(None)           # a reduced substep starts from the previous state

    fast = SW2Simulation(case, opts=opts_fast)
    warm = [fast.advance(before_attempt=guess_hook) for _ in range(W)]   # spin-up, graphs, AMG set-up
    state0 = fast.state()
    t0 = fast.t
    hold0 = (fast.dt_hold, fast.hold_count)     # step control carried into the timed window
    plain = None
    if not args.no_plain:
        plain = SW2Simulation(case, opts=opts_plain)
        plain.model.load_state(*state0[:3], bc_mask=state0[3])
        plain.t = t0
        plain.advance()                         # builds its hierarchy / graphs
        plain.model.load_state(*state0[:3], bc_mask=state0[3])
        plain.t = t0
        plain.dt_hold, plain.hold_count = hold0

    def timed(sim, hook):
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        recs = []
        sim.start_mass_balance(1000.0)          # water density, kg/m^3
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()
        sim.model.set_profiling(True)
        sim.model.reset_profile()
        s = torch.cuda.ExternalStream(sim.model.stream)
        ev0.record(s)
        for _ in range(K):
            recs.append(sim.advance(before_attempt=hook))
        ev1.record(s)
        torch.cuda.synchronize()
        ms = ev0.elapsed_time(ev1)
        prof_ms, prof_n = sim.model.profile()
        sim.model.set_profiling(False)
        if dist is not None:
            ms = max_over_ranks(ms, dist)
            dist.barrier()
        return ms, recs, prof_ms, prof_n

    with ClockSampler(local) as clk:
        ms_fast, rec_fast, prof_ms, prof_n = timed(fast, guess_hook)
    clocks = clk.summary()
    ms_plain, rec_plain = None, None
    if plain is not None:
        ms_plain, rec_plain, _, _ = timed(plain, None)
    fast_final = fast.state()[0]
    plain_err = rel_errors(fast_final, plain.state()[0]) if plain is not None else None

    # roofline of the dominant kernel of the fast path: the FP32 AMG smoothing sweep
    rf_ms, rf_bytes = fast.model.time_kernel(5, 20)
    spmv_ms, spmv_bytes = fast.model.time_kernel(0, 20)
    fd_ms, fd_bytes = fast.model.time_kernel(1, 5)
    # one FP32 GMRES iteration of the fast path, by part (CUDA events on the model's stream)
    breakdown = None
    try:
        cyc_ms, cyc_its = fast.model.time_kernel(8, 3)
        vc_ms, _ = fast.model.time_kernel(6, 10)
        sp32_ms, _ = fast.model.time_kernel(7, 20)
        pc_ms, pc_bytes = fast.model.time_kernel(9, 20)
        it_ms = cyc_ms / max(cyc_its, 1.0)
        breakdown = {"iteration_ms": it_ms, "amg_vcycle_ms": vc_ms, "of_which_level0_sweeps_ms": 4 * rf_ms,
                     "of_which_chunk_correction_ms": pc_ms, "spmv_ms": sp32_ms,
                     "gram_schmidt_and_vector_ops_ms": it_ms - vc_ms - sp32_ms, "cycle_iterations": cyc_its,
                     "chunk_correction_bytes": pc_bytes}
    except Exception as e:  # noqa: BLE001 - reported, not fatal
        breakdown = {"error": str(e)}
    peaks = {}
    try:
        with open(os.path.join(HERE, "MEASURED_PEAKS.json")) as fh:
            peaks = json.load(fh)
    except OSError:
        pass
    hbm = float(peaks.get("hbm_gbs", 0) or 0)
    peak_src = "measured"
    if hbm <= 0:
        hbm, peak_src = 6650.0, "fallback"
    achieved = rf_bytes / (rf_ms * 1e-3) / 1e9
    traffic = None
    tfile = os.path.join(HERE, "profiles", "traffic.json")
    if os.path.exists(tfile):
        try:
            with open(tfile) as fh:
                traffic = json.load(fh).get("amg_smooth_fp32_bytes_per_launch")
        except (OSError, ValueError):
            traffic = None

    # end to end through the reference-facing C ABI with host buffers (sw2g_fe_newton per
    # solve, pinned buffers), with the same dt reduction on a failed solve as advance()
    e2e = None
    if not args.no_e2e:
        m = fast.model
        n = m.ndofs
        sol_h = torch.empty(n, dtype=torch.float64, pin_memory=True)
        old_h = torch.empty(n, dtype=torch.float64, pin_memory=True)
        older_h = torch.empty(n, dtype=torch.float64, pin_memory=True)
        mask_h = torch.empty(n, dtype=torch.int32, pin_memory=True)
        dir_h = torch.zeros(n, dtype=torch.float64, pin_memory=True)
        s, so, soo, mk = state0
        old_h.numpy()[:] = s; older_h.numpy()[:] = so; mask_h.numpy()[:] = mk
        st = NewtonStats()
        L = lib()
        solves = 0

        o_e2e = [opts_fast]

        def solve(t_start, h):
            nonlocal solves
            d, vx, vy = fast.bc_values(t_start, t_start + h)
            m.set_step(h, d, vx, vy)
            if guesser is not None and h == case.dt:
                guesser.predict_host(m, old_h.numpy(), older_h.numpy())
            elif guesser is not None:
                m.set_guess(None)
            rc = L.sw2g_fe_newton(m.h, C.c_void_p(sol_h.data_ptr()), C.c_void_p(old_h.data_ptr()),
                                  C.c_void_p(older_h.data_ptr()), C.c_void_p(mask_h.data_ptr()),
                                  C.c_void_p(dir_h.data_ptr()), C.byref(o_e2e[0]), C.byref(st))
            solves += 1
            if rc not in (0, -5):                 # -5: non-finite residual, a failed solve (state kept)
                raise RuntimeError(L.sw2g_last_error().decode())
            if rc == 0 and st.success:
                older_h.numpy()[:] = old_h.numpy(); old_h.numpy()[:] = sol_h.numpy()
                return True
            return False

        t_e = t0
        e2e_ok = 0
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()
        w0 = time.perf_counter()
        hold, hold_n = hold0                    # the same step control as advance()
        for _ in range(K):
            target = t_e + case.dt
            held = hold is not None and hold < case.dt
            h = hold if held else case.dt
            o_e2e[0] = opts_fast
            if held and opts_fast.tol_nonlin_rel > 0:
                o_e2e[0] = type(opts_fast).from_buffer_copy(opts_fast)
                o_e2e[0].tol_nonlin_rel = opts_fast.tol_nonlin_rel * case.dt / h
            first, cuts, ok = True, 0, True
            while t_e + 1e-6 * case.dt < target:
                hh = min(h, target - t_e)
                good = solve(t_e, hh)
                if first and (held or not good) and st.tol_used > 0 and opts_fast.tol_nonlin_rel > 0:
                    # shorter steps keep the interval's tolerance, as advance() does
                    o_e2e[0] = type(opts_fast).from_buffer_copy(opts_fast)
                    o_e2e[0].tol_nonlin_min = st.tol_used
                first = False
                if good:
                    t_e += hh
                    continue
                cuts += 1
                if cuts > 3:
                    ok = False
                    break
                h *= DT_REDUCE_FACTOR
            if ok and fast.keep_reduced_dt > 0:
                if cuts:
                    hold, hold_n = h, 0
                elif held:
                    hold_n += 1
                    if hold_n >= fast.keep_reduced_dt:
                        grown = h / DT_REDUCE_FACTOR
                        hold, hold_n = (None if grown >= case.dt * (1 - 1e-12) else grown), 0
            e2e_ok += int(ok)
        wall = time.perf_counter() - w0
        wall = max_over_ranks(wall, dist)
        e2e = {"value": world * e2e_ok / wall, "unit": UNIT,
               "h2d_bytes_per_step": 3 * 8 * n + 4 * n + 8 * n + (8 * n if guesser is not None else 0),
               "d2h_bytes_per_step": 8 * n + 4 * n, "intervals_ok": e2e_ok, "solves": solves,
               "api": "sw2g_fe_newton (host buffers, pinned), the step control of advance()"}

    # the reference's CPU run on the sample (rank 0): timing and the final state, and our two
    # paths on the same sample with the same options, compared with it
    sample_err = None
    if cpu_run is not None:
        try:
            scase, srun = cpu_run
            value_cpu, _, sample, ref_final = cpu_reference_result(srun, scase, W)
            cpu = {"value": value_cpu, "unit": UNIT, "cores": 1, "kind": "reference", "sample": sample}
            if ref_final is not None:
                sample_err = {}
                for name, o in (("fast", opts_fast), ("plain", opts_plain)):
                    ss = SW2Simulation(scase, opts=o)
                    recs = [ss.advance() for _ in range(W + K)]
                    sample_err[name] = {"rel_err_hu_v": rel_errors(ss.state()[0], ref_final),
                                        "intervals_ok": sum(r["success"] for r in recs),
                                        "dt_cuts": sum(r["dt_cuts"] for r in recs)}
                    ss.model.close()
                sample_err["steps"] = W + K
                sample_err["note"] = ("state after the same steps as the reference's run; the reference applies "
                                      "its absolute Newton test 1e-8, ours the relative one")
        except Exception as e:  # noqa: BLE001
            cpu = cpu_baseline_failed(e)

    if rank != 0:
        _cleanup(fast, plain, guesser)
        if dist is not None:
            dist.destroy_process_group()
        return
    sf = interval_summary(rec_fast)
    names = ["residual", "fd_jacobian", "jacobian_gather", "prepare_precond_setup", "krylov", "other"]
    sf.update({"guess_used": [r.get("guess_used", 0) for r in rec_fast],
               "prev_resid": [r.get("prev_resid_max") for r in rec_fast],
               "class_ms": dict(zip(names, [round(float(x), 2) for x in prof_ms])),
               "mass_balance": fast.mass_balance(),
               "warmup_intervals_ok": sum(r["success"] for r in warm)})
    out = {
        "metric": METRIC, "value": world * sf["intervals_ok"] / (ms_fast * 1e-3), "unit": UNIT, "n_gpus": world,
        "steps": K, "warmup": W, "ms_per_step": ms_fast / K, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64+f32", "data": "synthetic",
        "config": {"workload": args.workload, "ntri": case.ntri, "nnodes": case.nnodes, "ndofs": 3 * case.nnodes,
                   "nnz": fast.model.nnz, "dt_s": case.dt, "tol_nonlin": 1e-8, "tol_nonlin_rel": args.tol_rel,
                   "krylov": f"GMRES({args.restart})+AMG", "krylov_forcing": args.krylov_tol,
                   "guess": args.guess if guesser is not None else "none",
                   "fast_precision": ("AMG preconditioner FP32, Krylov/residual/FD FP64" if args.basis == 64 else
                                      "GMRES cycle (basis, SpMV, AMG) FP32 inside FP64 refinement; residual/FD FP64"),
                   "step": "one dt interval (advance: a failed Newton solve is undone and the interval covered "
                           "at dt x 0.25; after a cut the next 4 intervals start at the reduced dt, then it grows "
                           "back by 4x; every solve meets the interval's Newton tolerance); value counts completed "
                           "intervals only",
                   "parallelism": f"replicas{world}", "l2": "inputs larger than L2 (1.5 GB matrix)"},
        "fast_detail": sf,
        "gpu_launches": int(np.sum(prof_n)),
        "clocks": clocks,
        "roofline": {"kernel": "k_tile_rows<1> (AMG level-0 smoothing sweep, FP32)", "bound": "hbm",
                     "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
                     "peak_source": peak_src, "traffic": traffic, "algorithmic_bytes": rf_bytes,
                     "avg_launch_ms": rf_ms,
                     "spmv_fp64": {"achieved": spmv_bytes / (spmv_ms * 1e-3) / 1e9, "avg_launch_ms": spmv_ms,
                                   "frac": spmv_bytes / (spmv_ms * 1e-3) / 1e9 / hbm},
                     "fd_jacobian": {"achieved_gbs": fd_bytes / (fd_ms * 1e-3) / 1e9, "avg_launch_ms": fd_ms},
                     "gmres_iteration_fp32": breakdown},
        "e2e": e2e,
        "cpu_baseline": cpu,
        "error_vs_reference_sample": sample_err,
    }
    if ms_plain is not None:
        sp_ = interval_summary(rec_plain)
        sp_["mass_balance"] = plain.mass_balance()
        sp_["value"] = world * sp_["intervals_ok"] / (ms_plain * 1e-3)
        sp_["ms_per_step"] = ms_plain / K
        out["plain_fp64"] = sp_
        out["fast_vs_plain_rel_err_hu_v"] = plain_err
        if sp_["value"] > 0:
            out["speedup_vs_plain_fp64"] = out["value"] / sp_["value"]
    print(json.dumps(out), flush=True)
    _cleanup(fast, plain, guesser)
    if dist is not None:
        dist.destroy_process_group()


def _cleanup(*objs):
    """Release device objects in a fixed order before interpreter shutdown."""
    import torch
    torch.cuda.synchronize()
    for o in objs:
        if o is None:
            continue
        model = getattr(o, "model", None)
        if model is not None:
            model.close()
    torch.cuda.synchronize()


def main():
    args = parse()
    world, rank, local, dist = dist_setup(args)
    if args.impl == "reference":
        run_reference(args, world, rank, dist)
        if dist is not None:
            dist.destroy_process_group()
        return
    run_ours(args, world, rank, local, dist)


if __name__ == "__main__":
    main()
