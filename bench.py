#!/usr/bin/env python
"""Throughput of aerocfd's residual-and-update iteration on B200.

Workload (the headline line): the turbulent flat plate with Spalart-Allmaras,
193 x 129 x 33 nodes as 8 blocks of 25 x 129 x 33 along x (851,400 nodes),
wall spacing 5e-6 (y+ about 1 at Re_L 5e6), wall-normal ratio 1.1,
leading-edge clustering, M 0.2, Re_L 5e6, nu_t,inf = 3 nu_inf, CFL 5,
synthetic and generated in-process, started from freestream.  Scheme: the
reference's Roe flux on WENO3 states, 2nd-order central viscous terms, the
1st-order implicit LU-SGS update and the SA model with its scalar LU-SGS,
FP64 (the reference's arithmetic).

A step is one iteration of main.f90:343-447 for every block plus the residual
norm of sub_output_residual.f90 (the reference computes it every iteration).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

value: Mcell-iter/s (nodes x steps / device time), inputs resident on the GPU,
L2 flushed before every timed step (the case's arrays, 1.5 GB, exceed L2 as
well).  e2e: the same metric through the C-ABI with the solution (q and nu_t)
held on the host: every step copies them host->device, runs the iteration and
copies them and the residual back.  --impl reference times the CPU
restatement of the reference's algorithm (the reference is Fortran + MPI and
cannot be compiled in this image) on the host cores, one thread per block
like one MPI rank per block.

The last line of stdout is the one JSON line, the headline metric and what
qualifies it; a line `details: {...}` before it repeats that and adds the extra
objects: `tuning`, `kernels`, `iteration_roofline`, `mixed` (the device-timed metric with
aero_set_precision(1), and the mixed solution's max / L2 error against FP64
after 50 iterations from one state), `naca` (the laminar NACA0012 O-grid
4 x 129 x 65 x 3, M 0.5, Re 5000, AoA 2, CFL 2: the same measurements, its own
roofline, e2e and CPU sample), `convergence` (wall time to each drop milestone
1e-3 .. 1e-8 of the density residual on the 97x49x5 Euler bump channel with
the reference's Roe + WENO3 and with Steger-Warming + WENO5, FP64 and mixed),
`batched` (64 bump channels of uneven size in one batch, mixed precision,
CUDA-graph replay, autotuned launch shapes, against the same 64 cases run one
after another, with its error against an FP64 run of the same batch),
`schemes`, `sa_plate` (3000 iterations of the headline case from freestream
in FP64 and mixed: residual drop and skin-friction error) and `warm_start`.
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

WORKLOAD = "sa_flat_plate_193x129x33_8blocks_m0.2_re5e6_cfl5_fp64"
NACA_WORKLOAD = "naca0012_ogrid_4x129x65x3_laminar_fp64"
HBM_FALLBACK = 6650.0

# Algorithmic bytes per processed node of each kernel class (FP64): every
# array the kernel must read once plus every array it must write once (the
# LU-SGS records and other scratch a kernel writes for a later one are not
# credited).
KERNEL_BYTES = {
    "k_lusgs_sweep": 49 * 8,   # q,dxidx,inv_j,ra,rb,rc,diag,rhs read; dq*,dq w+r; q w
    "k_inviscid": 20 * 8,      # q,dxidx,inv_j read; rhsi write
    "k_viscous_a": 30 * 8,     # pri(u,v,w,t),amu2,dxidx,inv_j read; amu1,amu3,vor,fv/gv/hv write
    "k_viscous_b": 17 * 8,     # fv/gv/hv read; rhsv write
    "k_find_dt": 23 * 8,       # dxidx,pri(d,u,v,w,c),amu3 read; dt write
    "k_lusgs_prep": 22 * 8,    # pri(u,v,w,c),dxidx,dt,rhsi,rhsv read; ra,rb,rc,diag,rhs write
    "k_lusgs_mats": 24 * 8,    # q,dxidx,inv_j,ra,rb,rc,rhs,diag read (the blocks or records it writes are workspace)
    "k_getpri": 12 * 8,        # q read; pri write
    "k_sa_sweep": 21 * 8,      # pri(u,v,w),dxidx,inv_j,nut,dt,sa_rhs,diag read; dnut* w+r; dnut w; nut w
    "k_sa_a": 19 * 8,          # pri(u,v,w),dxidx,inv_j,nut,vor,length read; sa_rhs write (+ its source terms)
}
# The node box each kernel class runs over.
KERNEL_BOX = {"k_lusgs_sweep": "box1", "k_inviscid": "box1", "k_viscous_a": "box0", "k_viscous_b": "box0",
              "k_residual_partial": "box1", "k_lusgs_mats": "box1", "k_sa_sweep": "box1", "k_sa_a": "box1"}
# DRAM bytes (read + write) per launch of the dominant kernel of each
# workload, from one ncu capture of it (cold cache under replay), on 8 CTAs a
# block, which the autotuner chooses for both.
KERNEL_TRAFFIC = {(WORKLOAD, "k_lusgs_sweep"): 432.0e6 + 64.4e6,
                  (NACA_WORKLOAD, "k_lusgs_sweep"): 11.04e6}
# The whole iteration's compulsory footprint (FP64): read q, dxidx, inv_j,
# write q, dq* write+read = 30 words per node; SA adds nut r/w, dist, the
# alpha/beta/gamma tensors and dnut* w/r = 44 words.
ITER_BYTES = 240
ITER_BYTES_SA = 352


def init_replicas(world: int, local: int, backend: str = "nccl"):
    """One process per GPU (torchrun): the process group used only for the
    barrier around the timed region and the max over ranks; None at N = 1."""
    if world <= 1:
        return None
    import datetime
    import torch
    import torch.distributed as dist
    dist.init_process_group(backend, timeout=datetime.timedelta(seconds=120))
    if backend == "nccl":
        torch.cuda.set_device(local)
    return dist


def max_over_ranks(x: float, dist) -> float:
    """The largest value of x over the ranks (the job's time is its slowest
    replica's); x itself without a process group."""
    if dist is None:
        return x
    import torch
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], device=dev, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_rate(nodes: int, steps: int, world: int, seconds: float) -> float:
    """Mcell-iter/s of the whole job: every replica advances `nodes` nodes
    `steps` times in `seconds` (the max over ranks)."""
    return nodes * steps * world / seconds / 1e6


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--cpu-sample-seconds", type=float, default=12.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-converge", action="store_true", help="skip the time-to-1e-8 runs")
    ap.add_argument("--no-batch", action="store_true", help="skip the 64-case batch")
    ap.add_argument("--batch-split", action="store_true",
                    help="at N > 1, also split the 64-case batch over the ranks by whole cases")
    ap.add_argument("--no-warm-start", action="store_true", help="skip the learned warm start")
    ap.add_argument("--no-plate", action="store_true", help="skip the plate's 3000-iteration runs")
    ap.add_argument("--no-schemes", action="store_true", help="skip the WENO5 / WCNS5 workloads")
    ap.add_argument("--no-naca", action="store_true", help="skip the NACA0012 O-grid workload")
    return ap.parse_args()


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return HBM_FALLBACK, "fallback"


def make_case():
    """The headline workload: the SA flat plate, 8 blocks of 25 x 129 x 33."""
    from aerocfd_b200 import grids
    from aerocfd_b200.case import Config, IFLAG_NSSOLVER
    cfg = Config(solver=IFLAG_NSSOLVER, turbulence=2, ma=0.2, re=5.0e6, cfl=5.0, nutinf=3.0)
    return grids.flat_plate(nbi=8, nbj=1, nbk=1, cfg=cfg)


def make_naca():
    """The laminar NACA0012 O-grid 4 x 129 x 65 x 3 (M 0.5, Re 5000, AoA 2,
    CFL 2)."""
    from aerocfd_b200 import grids
    return grids.naca_ogrid()


CONV_WORKLOAD = "bump_channel_97x49x5_euler_m0.5_cfl5"
CONV_TARGET = 1e-8
CONV_MILESTONES = (1e-3, 1e-4, 1e-5, 1e-6, 1e-7, 1e-8)


def make_bump(inviscid: int = 4):
    """BASELINE config 1's channel and flow: 97 x 49 x 5, Euler, M 0.5, CFL 5;
    inviscid 4 = the reference's Roe + WENO3, 5 = Steger-Warming + WENO5."""
    from aerocfd_b200 import grids
    from aerocfd_b200.case import Config, IFLAG_EULERSOLVER
    return grids.bump_channel(cfg=Config(solver=IFLAG_EULERSOLVER, ma=0.5, re=1.0e6, cfl=5.0, inviscid=inviscid))


def converge_gpu(solver, mixed: bool, inviscid: int = 4, chunk: int = 500, its: int = 20000):
    """Wall time to each drop milestone of the density residual (relative to
    iteration 1) on the Euler bump channel, freestream start, over `its`
    iterations; the time to a milestone is the run's time per iteration times
    the iteration that first reached it."""
    import torch
    case = make_bump(inviscid)
    gc = solver.GpuCase(case)
    try:
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        gc.set_precision(mixed)
        gc.use_graphs(True)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        hs = [gc.step(chunk) for _ in range(its // chunk)]
        el = time.perf_counter() - t0
        status = gc.status()
    finally:
        gc.close()
    d = np.concatenate(hs)[:, 0]
    d = d / d[0]
    first = {}
    for m in CONV_MILESTONES:
        hit = np.nonzero(d <= m)[0]
        first[f"{m:.0e}"] = int(hit[0]) + 1 if len(hit) else None
    per_it = el / len(d)
    # where the history stops falling: the best drop and the iteration of it
    return {"iterations_run": len(d), "wall_s_run": el, "final_drop": float(d[-1]), "min_drop": float(d.min()),
            "iteration_of_min_drop": int(np.argmin(d)) + 1,
            "iterations_to": first,
            "wall_s_to": {k: (v * per_it if v else None) for k, v in first.items()},
            "device_status": status}


BATCH_WORKLOAD = "bump_batch_64_uneven_euler_mixed"


def profile_kernels(L, steps: int):
    """Per-kernel-class device time of `steps` steps (aero_profile: CUDA events
    around every launch on the stream it is launched on), with each class's
    share of the summed kernel time."""
    ms = ctypes.c_double(0.0)
    from aerocfd_b200 import _lib
    L.aero_profile(ctypes.c_int(1))
    _lib.check(L.aero_step_timed(ctypes.c_int(steps), ctypes.c_int(1), ctypes.byref(ms)), "profile")
    L.aero_profile(ctypes.c_int(0))
    kms = (ctypes.c_double * 32)()
    kct = (ctypes.c_longlong * 32)()
    nk = L.aero_profile_read(kms, kct, ctypes.c_int(32))
    L.aero_profile_name.restype = ctypes.c_char_p
    kernels = {}
    for i in range(nk):
        if kct[i]:
            kernels[L.aero_profile_name(ctypes.c_int(i)).decode()] = {"ms_total": kms[i], "launches": int(kct[i])}
    tot = max(1e-12, sum(x["ms_total"] for x in kernels.values()))
    for k in kernels:
        kernels[k]["share"] = kernels[k]["ms_total"] / tot
    return kernels, ms.value / steps


def box_nodes(case, boxname: str) -> int:
    tot = 0
    for b in case.blocks:
        bx = getattr(b, boxname)
        tot += (bx[1] - bx[0] + 1) * (bx[3] - bx[2] + 1) * (bx[5] - bx[4] + 1)
    return tot


def roofline_of(case, kernels, workload: str):
    """The dominant kernel class's achieved HBM rate: its algorithmic bytes
    per launch (KERNEL_BYTES x the nodes it runs over) / its event-timed
    average launch duration, against the measured copy bandwidth."""
    hbm, hbm_kind = peaks()
    dom = max(kernels, key=lambda k: kernels[k]["ms_total"])
    per_launch_ms = kernels[dom]["ms_total"] / kernels[dom]["launches"]
    n_units = box_nodes(case, KERNEL_BOX.get(dom, "box"))
    alg_bytes = KERNEL_BYTES.get(dom, ITER_BYTES) * n_units
    achieved = alg_bytes / (per_launch_ms / 1e3) / 1e9
    return {"bound": "hbm", "kernel": dom, "achieved": achieved, "peak": hbm, "unit": "GB/s",
            "frac": achieved / hbm, "peak_kind": hbm_kind, "traffic": KERNEL_TRAFFIC.get((workload, dom)),
            "alg_bytes_per_launch": alg_bytes, "units_per_launch": n_units,
            "bytes_per_unit": KERNEL_BYTES.get(dom, ITER_BYTES), "ms_per_launch": per_launch_ms}


def snapshot(case):
    return [{k: v.copy() for k, v in b.fields.items()} for b in case.blocks]


def restore(gc, case, snap, solver):
    for b, sn in zip(case.blocks, snap):
        for k, v in sn.items():
            b.fields[k][...] = v
    gc.sync_to_device(solver.ALL)


def mixed_error(gc, case, solver, its: int = 50):
    """Max and L2 error of the mixed-precision solution against FP64 after
    `its` iterations from the same state (q, and nu_t with SA), and of the
    density residual at the last of them; the FP64 mode is left set."""
    names = ("q", "nut") if case.cfg.turbulence else ("q",)
    gc.set_precision(False)
    gc.sync_to_host(solver.ALL)
    snap = snapshot(case)
    h64 = gc.step(its)
    gc.sync_to_host(solver.mask(*names))
    ref = {k: np.concatenate([b.fields[k].ravel().copy() for b in case.blocks]) for k in names}
    restore(gc, case, snap, solver)
    gc.set_precision(True)
    hmx = gc.step(its)
    gc.set_precision(False)
    gc.sync_to_host(solver.mask(*names))
    out = {"iterations": its}
    for k in names:
        got = np.concatenate([b.fields[k].ravel() for b in case.blocks])
        d = got - ref[k]
        out[f"{k}_max_rel"] = float(np.max(np.abs(d)) / np.max(np.abs(ref[k])))
        out[f"{k}_l2_rel"] = float(np.linalg.norm(d) / np.linalg.norm(ref[k]))
    out["resid_rho_rel"] = float(abs(hmx[-1, 0] - h64[-1, 0]) / abs(h64[-1, 0]))
    restore(gc, case, snap, solver)
    return out


def batched_gpu(solver, steps: int, warmup: int):
    """64 bump channels of uneven size (seed 0: ni ~ U{65..257}, nj ~ U{33..97},
    nk = 5, h ~ U[0.05,0.12], M ~ U[0.3,0.7]), mixed precision, as one batch
    with CUDA-graph replay and autotuned launch shapes, against the same cases
    run one after another with the same settings, and the same batch in FP64.
    Device time, L2 flushed before every timed step."""
    import torch
    from aerocfd_b200 import _lib, grids
    cases = grids.bump_batch(64, seed=0)
    nodes = sum(c.nodes for c in cases)
    batch, params = grids.batch_case(cases)
    gc = solver.GpuCase(batch, block_params=params)
    ms = ctypes.c_double(0.0)
    out = {"workload": BATCH_WORKLOAD, "cases": 64, "nodes": nodes, "steps": steps}
    try:
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        gc.set_precision(True)
        out["tuning"] = gc.autotune(3)
        gc.use_graphs(True)
        for mixed in (True, False):
            gc.set_precision(mixed)
            gc.step(warmup, history=False)
            torch.cuda.synchronize()
            _lib.check(gc.L.aero_step_timed(ctypes.c_int(steps), ctypes.c_int(1), ctypes.byref(ms)), "batch timed")
            if mixed:
                batch_s = ms.value / 1e3
                out.update({"value": nodes * steps / batch_s / 1e6, "unit": "Mcell-iter/s",
                            "ms_per_step": 1e3 * batch_s / steps})
            else:
                out["fp64"] = {"value": nodes * steps / (ms.value / 1e3) / 1e6, "ms_per_step": ms.value / steps}
        gc.set_precision(True)
        kernels, step_ms = profile_kernels(gc.L, max(5, steps // 2))
        out["kernels"] = kernels
        out["roofline"] = roofline_of(batch, kernels, BATCH_WORKLOAD)
        out["iteration_roofline"] = {"bytes_per_node_iter": ITER_BYTES,
                                     "achieved_gbs": ITER_BYTES * nodes / (out["ms_per_step"] / 1e3) / 1e9,
                                     "frac": ITER_BYTES * nodes / (out["ms_per_step"] / 1e3) / 1e9 / peaks()[0]}
        out["error_vs_fp64"] = mixed_error(gc, batch, solver, 50)
        out["device_status"] = gc.status()
    finally:
        gc.close()
    seq_s = 0.0
    for c in grids.bump_batch(64, seed=0):
        g1 = solver.GpuCase(c)
        try:
            g1.compute_geometry()
            g1.init_flowfield()
            g1.start()
            g1.set_precision(True)
            g1.use_graphs(True)
            g1.step(warmup, history=False)
            _lib.check(g1.L.aero_step_timed(ctypes.c_int(steps), ctypes.c_int(1), ctypes.byref(ms)), "case timed")
            seq_s += ms.value / 1e3
        finally:
            g1.close()
    out.update({"sequential_value": nodes * steps / seq_s / 1e6, "sequential_ms_per_step": 1e3 * seq_s / steps,
                "speedup_vs_sequential": seq_s / batch_s,
                "note": "one launch per kernel for all 64 cases, each step replayed from a CUDA graph; "
                        "sequential = the 64 cases one after another, same settings, device time summed"})
    return out


PLATE_WORKLOAD = "sa_flat_plate_193x129x33_8blocks_m0.2_re5e6_cfl5"


def plate_cf(case) -> np.ndarray:
    """Skin friction on the wall nodes of the middle k-plane, i in order:
    cf = 2 mu_w u_t / dn / re (rho = u = 1), the wall-shear term of
    clcd_output with the first off-wall node (host arrays)."""
    out = []
    for b in case.blocks:
        if not any(sf.face == 3 and sf.blk_t == -20 for sf in b.subfaces):
            continue
        k = (b.nk + 1) // 2
        is0, ie0 = b.box0[0], b.box0[1]
        for i in range(is0, ie0 + (1 if b is case.blocks[-1] else 0)):
            dn = np.sqrt(sum((b.at(c, 1, i, 2, k) - b.at(c, 1, i, 1, k)) ** 2 for c in ("x", "y", "z")))
            out.append(2.0 * b.at("amu", 3, i, 1, k) * b.at("pri_v", 2, i, 2, k) / dn / case.cfg.re)
    return np.array(out)


def batched_split_gpu(solver, steps: int, warmup: int, rank: int, world: int, dist):
    """At N > 1: the 64-case batch of ``batched_gpu`` split over the ranks by
    whole cases (longest-processing-time on node counts,
    aerocfd_b200/distribute.py), each rank's share one batch in mixed
    precision with CUDA-graph replay and its own autotuned launch shapes; no
    data moves between ranks.  The job's time is the slowest rank's device
    time (max over ranks), so `value` is the whole list's node updates per
    second: strong scaling over the fixed list."""
    import torch
    from aerocfd_b200 import _lib, distribute, grids
    cases = grids.bump_batch(64, seed=0)
    nodes = [c.nodes for c in cases]
    parts = distribute.assign(nodes, world)
    mine = [cases[i] for i in parts[rank]]
    batch, params = grids.batch_case(mine)
    gc = solver.GpuCase(batch, block_params=params)
    ms = ctypes.c_double(0.0)
    try:
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        gc.set_precision(True)
        gc.autotune(3)
        gc.use_graphs(True)
        gc.step(warmup, history=False)
        torch.cuda.synchronize()
        dist.barrier()
        _lib.check(gc.L.aero_step_timed(ctypes.c_int(steps), ctypes.c_int(1), ctypes.byref(ms)), "split timed")
        status = gc.status()
    finally:
        gc.close()
    t = max_over_ranks(ms.value / 1e3, dist)
    bad = max_over_ranks(float(status != 0), dist)
    total = sum(nodes)
    return {"workload": BATCH_WORKLOAD, "cases": len(cases), "nodes": total, "steps": steps,
            "value": total * steps / t / 1e6, "unit": "Mcell-iter/s", "ms_per_step": 1e3 * t / steps,
            "scaling": "strong", "split": "whole cases per rank, longest-processing-time on node counts",
            "rank_nodes": [sum(nodes[i] for i in p) for p in parts], "rank_cases": [len(p) for p in parts],
            "precision": "mixed", "any_rank_status_nonzero": bool(bad)}


def sa_plate_gpu(solver, its: int = 3000, chunk: int = 500):
    """The headline plate run from the freestream for `its` iterations in
    FP64 and in mixed precision (autotuned shapes, CUDA graphs): the residual
    drop of each, the wall time, and the skin friction of the mixed run
    against FP64 (the config's 1e-8 drop needs far more iterations than a
    bench run)."""
    import torch
    case = make_case()
    gc = solver.GpuCase(case)
    out = {"workload": PLATE_WORKLOAD, "blocks": len(case.blocks), "nodes": case.nodes}
    cf = {}
    try:
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        out["tuning"] = gc.autotune(3)
        gc.use_graphs(True)
        for mixed in (False, True):
            gc.init_flowfield()
            gc.start()
            gc.set_precision(mixed)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            h = np.concatenate([gc.step(chunk) for _ in range(its // chunk)])
            el = time.perf_counter() - t0
            d = h[:, 0] / h[0, 0]
            key = "mixed" if mixed else "fp64"
            out[key] = {"iterations_run": len(d), "wall_s_run": el, "final_drop": float(d[-1]),
                        "min_drop": float(d.min()), "nut_final_drop": float(h[-1, 5] / h[0, 5])}
            gc.sync_to_host(solver.ALL)
            cf[key] = plate_cf(case)
        out["device_status"] = gc.status()
    finally:
        gc.close()
    dcf = cf["mixed"] - cf["fp64"]
    out["cf_mixed_vs_fp64"] = {"max_abs_rel": float(np.max(np.abs(dcf)) / np.max(np.abs(cf["fp64"]))),
                               "l2_rel": float(np.linalg.norm(dcf) / np.linalg.norm(cf["fp64"])),
                               "wall_nodes": len(dcf), "cf_range_fp64": [float(cf["fp64"].min()),
                                                                         float(cf["fp64"].max())]}
    out["note"] = ("the 1e-8 drop is not reached: in FP64 at CFL 5 the density residual falls to 1e-6 after "
                   "about 164,000 iterations and levels off at 4.2e-8 after about 390,000 (783 s on one B200), "
                   "the nut residual stopping at 7.8e-5 from about 100,000 iterations on")
    return out


def schemes_gpu(solver, steps: int, warmup: int):
    """The scheme-named workloads: the Euler bump 97 x 49 x 5 with
    Steger-Warming + WENO5 (CFL 5, 500 iterations) and the laminar NACA0012
    O-grid 4 x 129 x 65 x 3 with WCNS5 + Roe (CFL 2, 3000 iterations), each
    beside the same case with the reference's Roe + WENO3: device-timed
    throughput (L2 flushed before every step), the density-residual drop over
    the run and, for the aerofoil, cl and cd at its end."""
    import torch
    from aerocfd_b200 import _lib, grids
    from aerocfd_b200.case import Config, IFLAG_EULERSOLVER, IFLAG_NSSOLVER, SCHEME_NAMES
    out = {}
    runs = [("bump_97x49x5_euler_m0.5_cfl5", 500,
             lambda inv: grids.bump_channel(cfg=Config(solver=IFLAG_EULERSOLVER, ma=0.5, re=1.0e6, cfl=5.0,
                                                       inviscid=inv)), (5, 4)),
            ("naca0012_ogrid_4x129x65x3_laminar", 3000,
             lambda inv: grids.naca_ogrid(cfg=Config(solver=IFLAG_NSSOLVER, ma=0.5, re=5000.0, aoa_deg=2.0, cfl=2.0,
                                                     inviscid=inv)), (8, 4))]
    ms = ctypes.c_double(0.0)
    for name, its, make, schemes in runs:
        res = {}
        for inv in schemes:
            case = make(inv)
            gc = solver.GpuCase(case)
            try:
                gc.compute_geometry()
                gc.init_flowfield()
                gc.start()
                gc.use_graphs(True)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                h = gc.step(its)
                el = time.perf_counter() - t0
                clcd = gc.clcd_output(1.0)[6:8] if inv != 5 else None
                gc.step(warmup, history=False)
                _lib.check(gc.L.aero_step_timed(ctypes.c_int(steps), ctypes.c_int(1), ctypes.byref(ms)), "scheme")
                r = {"value": case.nodes * steps / (ms.value / 1e3) / 1e6, "unit": "Mcell-iter/s",
                     "ms_per_step": ms.value / steps, "iterations": its, "wall_s": el,
                     "drop": float(h[-1, 0] / h[0, 0]), "device_status": gc.status()}
                if clcd is not None:
                    r["cl"], r["cd"] = float(clcd[0]), float(clcd[1])
                res[SCHEME_NAMES[inv]] = r
            finally:
                gc.close()
        out[name] = res
    out["note"] = "iflag_inviscid 5 and 8 have no code in the reference (it stops on them); FP64 here"
    return out


def warm_start_gpu(solver, n_train: int = 48, n_test: int = 8, ni: int = 97, nj: int = 49):
    """Learned warm start on the bump family (97 x 49 x 5, farfield channel,
    h ~ U[0.05,0.12], M ~ U[0.3,0.7]): training fields from n_train members run
    3000 iterations as one batch, an 8 x 256 BF16 MLP trained on them with the
    tcgen05 kernels, then n_test held-out members from freestream (cold) and
    from the prediction (warm), both as a batch, to a 1e-8 drop of the cold
    run's iteration-1 density residual; forces compared at the end."""
    from aerocfd_b200 import warmstart as W
    fam = W.family(n_train + n_test, seed=11, ni=ni, nj=nj, nk=5)
    train, test = fam[:n_train], fam[n_train:]
    t0 = time.perf_counter()
    _, gen_s, batch = W.run_batch(solver, train, 3000, chunk=500)
    X = np.concatenate([W.features(c, h, m) for c, h, m in train])
    T = np.concatenate([W.targets(W.member(batch, i, c.cfg)) for i, (c, h, m) in enumerate(train)])
    net = W.Network(width=256, depth=8, batch=8192, seed=3)
    try:
        t1 = time.perf_counter()
        loss = net.train(X, T, steps=4000, lr=1e-3)
        train_s = time.perf_counter() - t1
        warm = {i: net.predict(W.features(c, h, m)) for i, (c, h, m) in enumerate(test)}
    finally:
        net.close()
    iters, chunk = 6000, 50
    hc, cold_s, bc = W.run_batch(solver, test, iters, chunk=chunk)
    hw, warm_s, bw = W.run_batch(solver, test, iters, chunk=chunk, warm=warm)
    out = {"family": f"bump_farfield_{ni}x{nj}x5", "train_members": n_train, "test_members": n_test,
           "network": "8 x 256 SiLU MLP, BF16 weights/activations, FP32 accumulation, tcgen05 GEMMs",
           "samples": int(len(X)), "train_steps": 4000, "train_s": train_s, "data_generation_s": gen_s,
           "loss_first_last": [float(loss[:10].mean()), float(loss[-10:].mean())]}
    out["iterations_run"] = iters
    for drop in (1e-4, 1e-6, 1e-8):
        # every member is reported: the iteration at which it first reached
        # the level, or null when it did not within the run; the batch's wall
        # time to the level is the time until its slowest member reached it,
        # null unless every member did
        level = hc[0] * drop
        ic, iw = W.first_below(hc, level, chunk), W.first_below(hw, level, chunk)
        both = (ic > 0) & (iw > 0)
        out[f"{drop:.0e}"] = {
            "cold_iterations": [int(v) if v > 0 else None for v in ic],
            "warm_iterations": [int(v) if v > 0 else None for v in iw],
            "cold_members_reached": int((ic > 0).sum()), "warm_members_reached": int((iw > 0).sum()),
            "cold_iterations_mean_of_both_reached": float(ic[both].mean()) if both.any() else None,
            "warm_iterations_mean_of_both_reached": float(iw[both].mean()) if both.any() else None,
            "cold_wall_s_all_members": float(cold_s * ic.max() / iters) if (ic > 0).all() else None,
            "warm_wall_s_all_members": float(warm_s * iw.max() / iters) if (iw > 0).all() else None}
    out["iteration1_residual_ratio_warm_over_cold"] = float(np.mean(hw[0] / hc[0]))
    diffs = []
    for i, (c, h, m) in enumerate(test):
        fc = W.wall_force(solver, W.member(bc, i, c.cfg))
        fw = W.wall_force(solver, W.member(bw, i, c.cfg))
        diffs.append(float(np.max(np.abs(fw[[6, 7]] - fc[[6, 7]]) / np.abs(fc[[6, 7]]))))
    out["cl_cd_max_rel_diff"] = max(diffs)
    out["total_s"] = time.perf_counter() - t0
    return out


def warm_start_naca_gpu(solver, n_train: int = 48, n_test: int = 12, its_train: int = 3000, its_test: int = 3000,
                        chunk: int = 100):
    """Learned warm start on the NACA 4-digit family with SA (config 5's
    parameter ranges: t 8-15 %, camber 0-4 % at 0.2-0.6, AoA -2..6 deg,
    M 0.3-0.7, Re 1e6-1e7) on the 4-block O-grid 4 x 129 x 65 x 3 (wall
    spacing 5e-6, CFL 3): n_train members run its_train iterations as one
    batch give the training fields (members that fail, retired by their
    block status, are left out), an 8 x 256 BF16 MLP is trained on them
    with the tcgen05 kernels, and n_test held-out members run its_test
    iterations from the freestream (cold, FP64), from the prediction (warm,
    FP64) and from the prediction in mixed precision, each as one batch.
    Reported per member: the iteration at which the density residual first
    falls to each level (a drop relative to the cold run's iteration-1
    residual), the wall time for the whole batch to get there, and cl, cd of
    the cold and warm runs after its_test iterations."""
    from aerocfd_b200 import grids, warmstart as W
    fam = W.naca_family(n_train + n_test, seed=11)
    train, test = fam[:n_train], fam[n_train:]
    t0 = time.perf_counter()
    _, gen_s, batch, st_train = W.run_family_batch(solver, train, its_train, chunk=chunk)
    cases_tr = [c for c, _ in train]
    ok = [i for i in range(n_train) if st_train[i] == 0]  # a member that failed gives no training data
    X = np.concatenate([W.naca_features(*train[i]) for i in ok])
    T = np.concatenate([W.naca_targets(grids.unbatch(batch, cases_tr, i)) for i in ok])
    del batch
    net = W.Network(n_in=W.NACA_IN, n_out=W.NACA_OUT, width=256, depth=8, batch=8192, seed=3)
    try:
        t1 = time.perf_counter()
        loss = net.train(X, T, steps=4000, lr=1e-3)
        train_s = time.perf_counter() - t1
        warm = {i: net.predict(W.naca_features(c, p)) for i, (c, p) in enumerate(test)}
    finally:
        net.close()
    runs = {"cold": W.run_family_batch(solver, test, its_test, chunk=chunk),
            "warm": W.run_family_batch(solver, test, its_test, chunk=chunk, warm=warm),
            "warm_mixed": W.run_family_batch(solver, test, its_test, chunk=chunk, warm=warm, mixed=True)}
    hc = runs["cold"][0]
    out = {"family": "naca4_sa_ogrid_4x129x65x3_cfl3", "train_members": n_train, "train_members_used": len(ok),
           "test_members": n_test,
           "iterations_train": its_train, "iterations_test": its_test,
           "network": "8 x 256 SiLU MLP, BF16 weights/activations, FP32 accumulation, tcgen05 GEMMs",
           "samples": int(len(X)), "train_steps": 4000, "train_s": train_s, "data_generation_s": gen_s,
           "loss_first_last": [float(loss[:10].mean()), float(loss[-10:].mean())],
           "iteration1_residual_ratio_warm_over_cold": float(np.mean(runs["warm"][0][0] / hc[0])),
           "member_status": {k: [int(x) for x in v[3]] for k, v in runs.items()}}
    levels = {}
    for drop in (1e-1, 1e-2, 1e-3):
        lv = hc[0] * drop
        row = {}
        for k, (h, wall, _, st) in runs.items():
            it = W.first_below(h, lv, chunk)
            it[st != 0] = -1  # a failed member is retired (its residual then reads 0): it reached nothing
            row[k] = {"iterations": [int(v) if v > 0 else None for v in it], "members_reached": int((it > 0).sum()),
                      "members_failed": int((st != 0).sum()),
                      "wall_s_all_members": float(wall * it.max() / its_test) if (it > 0).all() else None}
        # members that both the cold run and the warm run brought to the level
        both = [i for i in range(n_test) if row["cold"]["iterations"][i] and row["warm"]["iterations"][i]]
        row["mean_iterations_both_reached"] = {
            k: (float(np.mean([row[k]["iterations"][i] for i in both])) if both else None) for k in ("cold", "warm")}
        row["members_warm_faster"] = int(sum(row["warm"]["iterations"][i] < row["cold"]["iterations"][i] for i in both))
        row["members_both_reached"] = len(both)
        levels[f"{drop:.0e}"] = row
    out["levels"] = levels
    forces = []
    for i in range(n_test):
        fc = W.wall_force(solver, grids.unbatch(runs["cold"][2], [c for c, _ in test], i))
        fw = W.wall_force(solver, grids.unbatch(runs["warm"][2], [c for c, _ in test], i))
        forces.append({"cl_cold": float(fc[6]), "cl_warm": float(fw[6]), "cd_cold": float(fc[7]), "cd_warm": float(fw[7])})
    out["forces_after_test_iterations"] = forces
    out["total_s"] = time.perf_counter() - t0
    return out


def mlp_gemm_gpu():
    """The warm-start network's tcgen05 BF16 GEMM (C = A B^T, FP32
    accumulation) timed on its own: the network's layer shape (a batch of 8192
    rows through a 256-wide layer) and a large square one, against the
    measured cuBLAS BF16 peak (burst)."""
    from aerocfd_b200 import _lib
    L = _lib.load()
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            peak, kind = float(json.load(f)["bf16_tflops"]), "measured"
    except Exception:
        peak, kind = 1590.0, "fallback"
    out = {"peak_tflops": peak, "peak_kind": kind}
    for name, (m, n, k, reps) in {"layer_8192x256x256": (8192, 256, 256, 200),
                                  "square_8192": (8192, 8192, 8192, 10)}.items():
        ms = ctypes.c_double(0.0)
        _lib.check(L.aero_mlp_gemm_timed(ctypes.c_int(m), ctypes.c_int(n), ctypes.c_int(k), ctypes.c_int(reps),
                                         ctypes.byref(ms)), "aero_mlp_gemm_timed")
        tf = 2.0 * m * n * k / (ms.value / 1e3) / 1e12
        out[name] = {"m": m, "n": n, "k": k, "ms": ms.value, "tflops": tf, "frac": tf / peak}
    return out


def bump_cpu_to_drop(drop: float = 1e-3, chunk: int = 50, cap: int = 4000):
    """The CPU restatement (1 block, 1 thread, the platform libm) run on the
    bump case from the freestream until its density residual first falls to
    `drop` times its iteration-1 value (checked every `chunk` iterations, as
    the GPU runs): (iterations, wall seconds, iterations per second)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle  # CPU baseline only
    case = make_bump()
    oc = oracle.OracleCase(case, libm=True)
    oc.geometry()
    oc.init_flowfield()
    oc.start()
    t0 = time.perf_counter()
    h = oc.iterate(1, 1)
    first, n, hit = h[0, 0], 1, None
    while n < cap:
        h = oc.iterate(chunk, 1)
        n += chunk
        if h[-1, 0] <= drop * first:
            hit = n
            break
    wall = time.perf_counter() - t0
    return hit, wall, n / wall


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.path = tempfile.mktemp(suffix=".csv")
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            self.proc.wait()

    def summary(self):
        rows = []
        try:
            for line in open(self.path):
                p = [x.strip() for x in line.split(",")]
                if len(p) >= 9:
                    rows.append(p)
        except Exception:
            pass
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        reasons = set()
        for r in rows:
            for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), r[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(rows)}


def cpu_reference(make, seconds: float, steps: int = 0, warmup: int = 0):
    """Times the CPU restatement (oracle/, -O3, one thread per block, the
    reference's one MPI rank per block) on the case `make` builds."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle  # CPU baseline only
    case = make()
    oc = oracle.OracleCase(case, libm=True)
    oc.geometry()
    oc.init_flowfield()
    oc.start()
    threads = min(len(case.blocks), os.cpu_count() or 1)
    if warmup:
        oc.iterate(warmup, threads)
    t0 = time.perf_counter()
    n = 0
    while True:
        oc.iterate(1, threads)
        n += 1
        el = time.perf_counter() - t0
        if steps and n >= steps:
            break
        if not steps and (el >= seconds and n >= 2):
            break
    el = time.perf_counter() - t0
    return case.nodes * n / el / 1e6, n, el, threads


def measure(solver, case, workload: str, args, world: int, local: int, dist, clocks: bool = False):
    """Device-timed, profiled, mixed-precision and end-to-end measurements of
    one workload; returns the line's fields (value, ms_per_step, roofline,
    kernels, mixed, e2e, ...)."""
    import torch
    from aerocfd_b200 import _lib
    gc = solver.GpuCase(case, device=local)
    L = gc.L
    try:
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        tuning = gc.autotune(3)   # launch shapes only; the state is restored
        gc.use_graphs(True)       # every step replayed from one CUDA graph
        gc.step(args.warmup, history=False)

        # ---- device-timed steps (resident inputs, L2 flushed before each step)
        cnt0 = ctypes.c_ulonglong(0)
        L.aero_launch_count(ctypes.byref(cnt0))
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        ms = ctypes.c_double(0.0)
        clk = ClockSampler(local) if clocks else None
        if clk:
            clk.__enter__()
        try:
            _lib.check(L.aero_step_timed(ctypes.c_int(args.steps), ctypes.c_int(1), ctypes.byref(ms)),
                       "aero_step_timed")
            torch.cuda.synchronize()
        finally:
            if clk:
                clk.__exit__(None, None, None)
        cnt1 = ctypes.c_ulonglong(0)
        L.aero_launch_count(ctypes.byref(cnt1))
        dev_s = max_over_ranks(ms.value / 1e3, dist)
        nodes = case.nodes
        out = {"value": whole_job_rate(nodes, args.steps, world, dev_s), "ms_per_step": 1e3 * dev_s / args.steps,
               "gpu_launches": int(cnt1.value - cnt0.value), "tuning": tuning}
        if clk:
            out["clocks"] = clk.summary()

        # ---- per-kernel profile (separate pass) for the roofline
        kernels, _ = profile_kernels(L, max(5, min(args.steps, 20)))
        out["kernels"] = kernels
        out["roofline"] = roofline_of(case, kernels, workload)
        hbm = peaks()[0]
        ib = ITER_BYTES_SA if case.cfg.turbulence else ITER_BYTES
        gbs = ib * nodes / (dev_s / args.steps) / 1e9
        out["iteration_roofline"] = {"bytes_per_node_iter": ib, "achieved_gbs": gbs, "frac": gbs / hbm}

        # ---- mixed precision: device-timed throughput, and its error against
        # FP64 after the same iterations from the same state
        gc.set_precision(True)
        gc.step(3, history=False)
        torch.cuda.synchronize()
        _lib.check(L.aero_step_timed(ctypes.c_int(args.steps), ctypes.c_int(1), ctypes.byref(ms)), "mixed timed")
        mixed_s = max_over_ranks(ms.value / 1e3, dist)
        out["mixed"] = {
            "value": whole_job_rate(nodes, args.steps, world, mixed_s), "unit": "Mcell-iter/s",
            "ms_per_step": 1e3 * mixed_s / args.steps,
            "dtype": "f32 WENO corrections / Roe dissipation / viscous stresses / SA source, advection and "
                     "diffusion terms / stored LU-SGS off-diagonal blocks; f64 state, metrics, rhs, implicit "
                     "diagonals, sweep products, dt, residual",
            "error_vs_fp64": mixed_error(gc, case, solver, 50)}

        # ---- end-to-end through the C-ABI with the solution held on the host
        names = ("q", "nut") if case.cfg.turbulence else ("q",)
        mq = solver.mask(*names)
        sbytes = sum(b.fields[k].nbytes for b in case.blocks for k in names)
        gc.sync_to_host(mq)
        res = np.zeros(7)
        for _ in range(2):
            gc.sync_to_device(mq)
            gc.step(1)
            gc.sync_to_host(mq)
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            gc.sync_to_device(mq)
            _lib.check(L.aero_step(ctypes.c_int(1), res.ctypes.data_as(ctypes.c_void_p), None), "aero_step")
            gc.sync_to_host(mq)
        e2e_s = max_over_ranks(time.perf_counter() - t0, dist)
        out["e2e"] = {"value": whole_job_rate(nodes, args.steps, world, e2e_s), "unit": "Mcell-iter/s",
                      "h2d_bytes_per_step": sbytes, "d2h_bytes_per_step": sbytes + 56,
                      "fields": list(names)}
        out["device_status"] = gc.status()
    finally:
        gc.close()
    return out


# Keys of the one JSON line; the objects under them keep the keys named here.
HEADLINE = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches", "device_status", "roofline")
HEADLINE_PARTS = {"roofline": ("bound", "kernel", "achieved", "unit", "frac", "ms_per_launch")}


def headline(line: dict) -> dict:
    """What the last line of stdout holds of a full result: short enough
    (about 1.3 kB) to stay whole where only the end of the output is kept."""
    return {k: {p: line[k][p] for p in HEADLINE_PARTS[k]} if k in HEADLINE_PARTS else line[k]
            for k in HEADLINE if k in line}


def main():
    args = parse()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.warmup < 3:
        args.warmup = 3
    case = make_case()
    config = {"workload": WORKLOAD, "blocks": len(case.blocks), "nodes": case.nodes,
              "grid": "193x129x33 as 8 blocks of 25x129x33 along x, wall spacing 5e-6, ratio 1.1",
              "ma": case.cfg.ma, "re": case.cfg.re, "nutinf_over_nuinf": case.cfg.nutinf, "cfl": case.cfg.cfl,
              "scheme": "roe_weno3 + central viscous + spalart-allmaras + lu-sgs (reference path)"}

    if args.impl == "reference":
        if rank != 0:
            return 0
        v, n, el, thr = cpu_reference(make_case, 0.0, steps=args.steps, warmup=args.warmup)
        line = {"metric": "Mcell-iter/s", "value": v, "unit": "Mcell-iter/s", "n_gpus": args.gpus,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * el / n,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
                "data": "synthetic (analytic flat-plate grid, freestream start)", "impl": "reference",
                "config": config,
                "cpu_baseline": {"value": v, "unit": "Mcell-iter/s", "cores": thr, "kind": "port",
                                 "sample": f"{n} full iterations of the workload on {thr} threads "
                                           f"(one per block), C++ -O3 restatement with glibc's pow/exp"},
                "e2e": {"value": v, "unit": "Mcell-iter/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line))
        return 0

    dist = init_replicas(world, local)
    from aerocfd_b200 import solver
    m = measure(solver, case, WORKLOAD, args, world, local, dist, clocks=True)
    if m["device_status"]:
        print(f"warning: device status word {m['device_status']}", file=sys.stderr)
    config.update({"l2": "flushed (256 MiB write) before every timed step; the case's arrays exceed L2",
                   "execution": "each step replayed from a CUDA graph; launch shapes from the autotuner",
                   "parallelism": f"replicas x{world}"})
    line = {"metric": "Mcell-iter/s", "value": m.pop("value"), "unit": "Mcell-iter/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": m.pop("ms_per_step"),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (analytic flat-plate grid, freestream start)", "config": config}
    line.update(m)
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        v, n, el, thr = cpu_reference(make_case, args.cpu_sample_seconds)
        line["cpu_baseline"] = {"value": v, "unit": "Mcell-iter/s", "cores": thr, "kind": "port",
                                "sample": f"{n} full iterations of the same workload, {el:.1f} s, "
                                          f"{thr} threads (one per block), C++ -O3 restatement"}
    if world == 1 and not args.no_naca:
        naca = make_naca()
        nm = measure(solver, naca, NACA_WORKLOAD, args, world, local, dist)
        nm.update({"workload": NACA_WORKLOAD, "blocks": len(naca.blocks), "nodes": naca.nodes,
                   "unit": "Mcell-iter/s"})
        if not args.no_cpu_baseline:
            v, n, el, thr = cpu_reference(make_naca, args.cpu_sample_seconds / 2)
            nm["cpu_baseline"] = {"value": v, "unit": "Mcell-iter/s", "cores": thr, "kind": "port",
                                  "sample": f"{n} full iterations, {el:.1f} s, {thr} threads (one per block)"}
        line["naca"] = nm
    if world > 1 and args.batch_split:
        line["batched_split"] = batched_split_gpu(solver, max(5, min(args.steps, 20)), args.warmup, rank, world,
                                                  dist)
    if world == 1 and not args.no_batch:
        line["batched"] = batched_gpu(solver, max(5, min(args.steps, 20)), args.warmup)
    if world == 1 and not args.no_schemes:
        line["schemes"] = schemes_gpu(solver, max(5, min(args.steps, 20)), args.warmup)
    if world == 1 and not args.no_plate:
        line["sa_plate"] = sa_plate_gpu(solver)
    if world == 1 and not args.no_warm_start:
        line["warm_start"] = warm_start_gpu(solver)
        line["mlp_gemm"] = mlp_gemm_gpu()
        line["warm_start_naca_sa"] = warm_start_naca_gpu(solver)
    if world == 1 and not args.no_converge:
        conv = {"workload": CONV_WORKLOAD, "target_drop": CONV_TARGET,
                "roe_weno3": {"fp64": converge_gpu(solver, False, 4), "mixed": converge_gpu(solver, True, 4)},
                "sw_weno5": {"fp64": converge_gpu(solver, False, 5), "mixed": converge_gpu(solver, True, 5)}}
        if not args.no_cpu_baseline:
            hit, wall, rate = bump_cpu_to_drop(1e-3)
            conv["cpu_reference"] = {
                "measured_to_1e-03": {"iterations": hit, "wall_s": wall,
                                      "gpu_fp64_wall_s": conv["roe_weno3"]["fp64"]["wall_s_to"]["1e-03"]},
                "its_per_s": rate, "cores": 1, "kind": "port",
                "wall_s_to_est": {k: (v / rate if v else None)
                                  for k, v in conv["roe_weno3"]["fp64"]["iterations_to"].items()},
                "note": "the oracle (Roe + WENO3, glibc pow/exp) run from the freestream to a 1e-3 drop, "
                        "timed; deeper levels estimated as its measured iteration rate x the FP64 GPU "
                        "iteration counts (the FP64 path reproduces the oracle's iterates); 1 thread = the "
                        "reference's layout for a 1-block case"}
        line["convergence"] = conv
    if rank == 0:
        print("details: " + json.dumps(line))
        print(json.dumps(headline(line)))
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
