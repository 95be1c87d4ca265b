"""Benchmark of the B200 finite-volume step and its discrete adjoint.

    python bench.py --gpus N --steps K --warmup W [--impl ours|reference]

Headline (the metric named for this path): forward + adjoint cell-updates/s on the 1M-cell workload: 5 km x 5 km plane-and-runout terrain at 4.9 m (1024^2
cells), one 30 m x 100 m pile, 512 time steps, J = sum of h^2 dx dy over a 500 m x 500 m box at
the final step, gradients with respect to pile height, basal and internal friction, 32 HBM
checkpoints (binomial schedule).  One benchmark "step" is one whole forward + adjoint run over the
512-step horizon; value = cells x 512 x K / device seconds (max over ranks).  A cell-update is one
cell advanced one forward step and taken back through its adjoint step, recomputation included.

Both precisions run.  The FP32-split run is the headline value only when its errors against the
FP64 run are within 1e-5 relative L2 on the final state and 1e-4 on every gradient; otherwise the
plain FP64 run (bit-identical to the reference's step()) is, and the FP32-split figures are
reported beside it with their errors.

Also reported: the FP32-split errors against FP64 (final state, J, gradients, lambda^0),
the forward step alone on the 3.75M-cell adaptive workload (hill + noise, 3 piles, 4 materials),
the batched 512-member ensemble (forward + adjoint, 300 steps) against the same members run one
after another, per-kernel device times (tracing), the roofline of the dominant kernel, e2e
through the C ABI with pinned host buffers, clocks, and a CPU baseline.

Multi-GPU: the headline workload is one instance, so N > 1 runs N independent replicas (one per
rank, "weak" scaling, no data-path collective); the ensemble's members are split over the ranks
(size-balanced greedy partition) with one gather of the per-member results; barrier and max over
ranks stay.

--impl reference: the reference's own forward + adjoint compiled from its sources
(oracle/_ref/ref_harness, mode 'DAF1': step() with the driver's solution recording, then the dual
solver's update_dual_grid / calc_jacobian / calc_adjoint) on the same 1M-cell workload, timed on
this host, one step at a time; rank 0 only.  Its mesh comes from oracle/meshgen.py (numpy, equal
to the product's mesh builder bit for bit), so the process never loads libda_b200.so.  One
"step" of that arm is one forward step and its reverse step over all 1M cells (the metric's unit
of work); --warmup steps run forward first and are neither timed nor taken back.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

METRIC = "cell-updates/s fwd+adjoint, FP32-split & batched vs plain FP64 GPU at ≤1e-5 rel err"
HEADLINE_WORKLOAD = "inclined-plane 5km x 5km uniform 1024^2, 1 pile"
HORIZON = 512
SNAPSHOTS = 32
ENS_STEPS = 300
ENS_SNAPSHOTS = 32


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks sampled during the timed region (every 200 ms)."""

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,utilization.gpu,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.t.join(timeout=2)
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 10:
                continue
            try:
                util = float(f[4])
                s = float(f[1])
                smax = float(f[2])
            except ValueError:
                continue
            if util > 0:
                sm.append(s)
                for k, nm in enumerate(names):
                    if f[6 + k].lower().startswith("active"):
                        reasons.add(nm)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples_under_load": len(sm)}


def dist_init(impl: str = "ours"):
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1 and impl == "ours":
        import datetime

        import torch
        import torch.distributed as dist
        # each rank's collectives and barriers on its own GPU
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300), device_id=torch.device("cuda", local))
    return ws, rank, local


def allmax(x: float, ws: int, dev: int) -> float:
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=f"cuda:{dev}")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def allsum(x: float, ws: int, dev: int) -> float:
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=f"cuda:{dev}")
    dist.all_reduce(t, op=dist.ReduceOp.SUM)
    return float(t.item())


def barrier(ws: int, dev: int):
    if ws > 1:
        import torch
        import torch.distributed as dist
        dist.barrier(device_ids=[dev])
        torch.cuda.synchronize(dev)


def pinned(count: int) -> np.ndarray:
    """A float64 host array in page-locked memory (torch's pinned allocator)."""
    import torch
    return torch.empty(count, dtype=torch.float64, pin_memory=True).numpy()


def wet_counts(m, h) -> tuple[int, int]:
    """(cells with h >= GEOFLOW_TINY, cells that are wet or have a wet face neighbour)."""
    wet = h >= 1e-4
    act = wet.copy()
    for k in range(8):
        e = m.nbr[k]
        ok = e >= 0
        act[ok] |= wet[e[ok]]
    return int(wet.sum()), int(act.sum())


def bytes_per_cell_update(precision: str) -> dict:
    """Algorithmic HBM bytes of one cell through one step (each array the cell needs touched once;
    neighbour re-reads are halo traffic), the rule of the per-unit figures for this path with the
    arrays of the committed layout (csrc/da_internal.h), r = 8 (FP64) / 4 (FP32-split) bytes per real:
      forward:  state in 3r + state out 3r + g (3), d_gravity (2), curvature (2) 7r + material and
                boundary flags 2 + neighbour table 4 x int32 16 + cell sizes 2r (+ centres 2 x 8 in
                FP64, whose slopes take centre differences as the reference does) + what the
                coefficient phase writes and the update phase reads back: two depth slopes, two
                velocities, the wave speed 10r and the friction signs 2
      adjoint:  lambda in 3r + U 3r + the same statics, flags, neighbours, sizes (and centres) +
                branch byte 1 + lambda out 3r + the depth slopes' four derivatives, kept likewise 8r
    FP64: forward 236 B, adjoint 243 B; FP32-split: 120 B and 123 B.  (Without what is kept, the
    one-pass figures of the path: FP64 154 B, FP32-split 78 B per forward cell-update.)"""
    r = 8 if precision == "fp64" else 4
    xy = 16 if precision == "fp64" else 0
    statics = 7 * r + 2 + 16 + 2 * r + xy
    return {"forward": 6 * r + statics + 10 * r + 2, "adjoint": 9 * r + statics + 1 + 8 * r}


# the launches of reverse steps, which the trace counts together: runs of them (k_reverse_run; 31 of the
# headline's 32) and single ones (k_youturn)
REVERSE = "k_reverse_run + k_youturn"


def algorithmic_bytes(precision: str, n_act: float) -> dict:
    """Algorithmic bytes of one launch of each kernel per time step it covers, over the cells the
    step actually processes (n_act: wet cells and their face neighbours; tile culling leaves the
    others untouched): k_steps one forward step, REVERSE one reverse step (the replayed forward
    step and the adjoint step), a checkpoint copy the state of those cells each way."""
    b = bytes_per_cell_update(precision)
    r = 8 if precision == "fp64" else 4
    return {"k_steps": b["forward"] * n_act, REVERSE: (b["forward"] + b["adjoint"]) * n_act,
            "snapshot_copy": 2 * 3 * r * n_act}


# DRAM bytes (read + write) from the committed ncu captures (the headline traffic and the dense
# k_steps summaries under profiles/).  Sparse headline kernels: bytes per active cell and step of a
# launch captured in the steady flow (reverse steps: one k_reverse_run of
# the 23 steps of iterations 258 to 236 of the 512-step sweep, 4272 active cells per step on average;
# k_steps: one launch of 32 steps after 256, 4553 active cells per step on average), scaled by the active
# cells of the traced run; the dense case: bytes per time step of a 10-step launch with every cell wet.
TRAFFIC_PER_ACTIVE_CELL = {
    ("fp64", REVERSE): (5517056 + 96768) / (23 * 4271.6),
    ("fp32", REVERSE): (3655424 + 90112) / (23 * 4271.1),
    ("fp64", "k_steps"): (1583104 + 25600) / (32 * 4552.6),
}
TRAFFIC_DENSE_PER_STEP = {
    "fp32": (5.144393e9 + 1.404350e9) / 10,
    "fp64": (9.412916e9 + 2.800689e9) / 10,
}


def traffic_per_launch(precision: str, kernel: str, n_act: float, steps_per_launch: float):
    per = TRAFFIC_PER_ACTIVE_CELL.get((precision, kernel))
    return None if per is None else per * n_act * steps_per_launch


# resident memory of one reference harness process per cell of the headline mesh (5.4 GB for
# 1,048,576 cells, measured), for sizing how many run side by side
REF_RSS_BYTES_PER_CELL = 5200


REF_MAX_STEPS, REF_MAX_WARMUP = 8, 3


def reference_replicas(cells: int) -> int:
    """Harness processes to run side by side: one per usable host core, as long as their resident
    memory stays under half of what the host has available."""
    cores = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    avail = None
    try:
        for line in open("/proc/meminfo"):
            if line.startswith("MemAvailable:"):
                avail = int(line.split()[1]) * 1024
    except OSError:
        pass
    by_mem = cores if avail is None else int(0.5 * avail // (REF_RSS_BYTES_PER_CELL * cells))
    return max(1, min(cores, by_mem))


def reference_fwdadj(steps: int, warm: int, side: int = 1024, replicas: int = 1) -> dict:
    """The reference's own forward + adjoint on the headline workload, timed on this host: `warm`
    forward steps untimed, then `steps` forward steps with the driver's solution recording and
    their `steps` reverse steps of the dual solver, each timed (oracle/_ref/ref_harness, mode
    'DAF1'); the oracle's restatement when the harness is not built.  One cell-update is one cell
    advanced one forward step and taken back through its reverse step, as in the GPU arm.  The
    mesh comes from oracle/meshgen.py, so libda_b200.so is never loaded.  replicas > 1: that many
    harness processes at once, one per host core; the rate is their total work over the slowest
    one's timed seconds (the reference's own parallel form, domain decomposition over MPI ranks,
    needs an MPI library; concurrent replicas bound what that could reach on these cores from
    above, with no halo exchange)."""
    import oracle
    from discrete_adjoint_b200.inputs import WORKLOAD3_BOX
    from discrete_adjoint_b200.mesh import Mesh
    from discrete_adjoint_b200.solver import MatProps
    from oracle import meshgen
    m = Mesh(**meshgen.headline_mesh(side))
    mat = MatProps(intfrict_deg=30.0, bedfrict_deg=[20.0])
    if oracle.reference_available():
        r = oracle.run_reference_fwdadj(m, mat, warm + steps, warm, WORKLOAD3_BOX, replicas=replicas)
        fwd, rev = r["fwd_seconds"][warm:], r["rev_seconds"]
        per = r["replica_seconds"]
        kind = "reference"
        how = ("the reference's own step() + SolRec::record_solution, then update_dual_grid + "
               "calc_jacobian + calc_adjoint (compiled from its sources by oracle/ref_build.py)")
    else:
        fwd, rev = oracle.time_port_fwdadj(m, mat, warm, steps, WORKLOAD3_BOX)
        per = [float(np.sum(fwd) + np.sum(rev))]
        kind = "port"
        how = "the oracle's restatement of the reference's step() and dual-solver step"
    secs = max(per)
    nproc = len(per)
    threads = ("1 thread (the reference is single-rank MPI code with no threading)" if nproc == 1 else
               f"{nproc} harness processes side by side, one per host core, each single-threaded "
               "(the reference's own parallelism is MPI ranks; the rate is the processes' total work "
               "over the slowest one's timed seconds)")
    return {"value": nproc * m.n * steps / secs, "ms_per_step": 1e3 * secs / steps, "kind": kind, "cells": m.n,
            "cores": nproc, "fwd_s_per_step": float(np.mean(fwd)), "rev_s_per_step": float(np.mean(rev)),
            "sample": f"{steps} forward steps and their {steps} reverse steps of the {m.n}-cell workload "
                      f"(after {warm} untimed forward steps) through {how}; {threads}; wall time of each step"}


def run_reference_arm(args, ws, rank):
    if rank != 0:
        return
    from discrete_adjoint_b200.inputs import WORKLOAD3_BOX
    # a bounded sample: each forward + reverse step of the reference takes seconds per process,
    # so at most REF_MAX_STEPS timed steps after at most REF_MAX_WARMUP untimed ones
    r = reference_fwdadj(max(1, min(args.steps, REF_MAX_STEPS)), min(args.warmup, REF_MAX_WARMUP),
                         replicas=reference_replicas(1024 * 1024))
    v = r["value"]
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "cell-updates/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": r["ms_per_step"],
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": HEADLINE_WORKLOAD, "cells": r["cells"], "horizon": HORIZON,
                       "functional": "sum h^2 dx dy over box " + str(WORKLOAD3_BOX), "precision": "fp64",
                       "step": "one forward step and its reverse (adjoint) step over every cell",
                       "forward_s_per_step": r["fwd_s_per_step"], "reverse_s_per_step": r["rev_s_per_step"]},
            "cpu_baseline": {"value": v, "unit": "cell-updates/s", "cores": r["cores"], "kind": r["kind"],
                             "sample": r["sample"]},
            "e2e": {"value": v, "unit": "cell-updates/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def fwdadj(args, ws, local):
    from discrete_adjoint_b200 import GeoflowContext, TimeProps, _ffi, adjoint_run, inputs
    w = inputs.workload3()
    m = w.mesh
    box = inputs.WORKLOAD3_BOX
    out = {}

    def fresh(prec):
        c = GeoflowContext(w.mat, TimeProps(), precision=prec, device=local)
        c.upload_mesh(m)
        c.set_state(m.h0, m.hu0, m.hv0)
        return c

    sampler = ClockSampler(local)
    for name, prec in (("fp64", _ffi.DA_PREC_FP64), ("fp32", _ffi.DA_PREC_FP32_SPLIT)):
        c = fresh(prec)
        # launch shape of the step kernels picked by the autotuner on this workload
        tune = c.autotune(10)
        for _ in range(args.warmup):
            adjoint_run(c, box, HORIZON, SNAPSHOTS, m.dh0_dpile)
        if not args.no_clocks:
            sampler = ClockSampler(local)
            sampler.start()
            time.sleep(0.3)
        barrier(ws, local)
        ms = 0.0
        g = None
        for _ in range(args.steps):
            g = adjoint_run(c, box, HORIZON, SNAPSHOTS, m.dh0_dpile)
            ms += g.device_ms
        barrier(ws, local)
        if not args.no_clocks:
            t_end = time.time() + 1.0
            while time.time() < t_end:
                adjoint_run(c, box, HORIZON, SNAPSHOTS, m.dh0_dpile)
        ms = allmax(ms, ws, local)
        gl = adjoint_run(c, box, HORIZON, SNAPSHOTS, m.dh0_dpile, want_lambda0=True)
        res = {"ms": ms, "value": m.n * HORIZON * args.steps * ws / (ms * 1e-3), "grad": gl,
               "forward_steps": g.forward_steps, "launch_shape": {"blocks_per_sm": tune["best"][0],
                                                                   "grid": tune["best"][1]}}
        res["clocks"] = sampler.stop() if not args.no_clocks else {"sm_mhz": None, "sm_max_mhz": None,
                                                                     "reasons": ["not sampled"]}
        # per-kernel device times of one traced run
        c.set_tracing(True)
        adjoint_run(c, box, HORIZON, SNAPSHOTS, m.dh0_dpile)
        res["trace"] = {REVERSE if k == "k_youturn" else k: v for k, v in c.trace(with_steps=True).items()}
        c.set_tracing(False)
        # e2e through the C ABI with pinned host buffers: H2D of the initial state and the pile
        # derivative, the run, D2H of the gradients and lambda^0
        h0, hu0, hv0, lam_host = pinned(m.n), pinned(m.n), pinned(m.n), pinned(3 * m.n)
        h0[:], hu0[:], hv0[:] = m.h0, m.hu0, m.hv0
        dpile = pinned(m.dh0_dpile.size).reshape(m.dh0_dpile.shape)
        dpile[:] = m.dh0_dpile
        barrier(ws, local)
        t0 = time.perf_counter()
        for _ in range(args.e2e_steps):
            c.set_state(h0, hu0, hv0)
            c.set_time(0.0, 0)
            ge = adjoint_run(c, box, HORIZON, SNAPSHOTS, dpile, lambda0_out=lam_host)
        e2e_s = allmax(time.perf_counter() - t0, ws, local)
        res["e2e"] = {"value": m.n * HORIZON * args.e2e_steps * ws / e2e_s, "unit": "cell-updates/s",
                      "h2d_bytes_per_step": 3 * 8 * m.n + 8 * dpile.size, "d2h_bytes_per_step": 3 * 8 * m.n + 8 * 32,
                      "J_matches_device_run": bool(ge.J == gl.J)}
        # forward state after the horizon, for the depth / momentum errors
        c.set_state(h0, hu0, hv0)
        c.set_time(0.0, 0)
        c.run(HORIZON)
        res["state"] = c.get_state()
        out[name] = res
        c.close()
    # wet / active counts over the horizon (forward states sampled every 64 steps)
    c = fresh(_ffi.DA_PREC_FP64)
    wv_, av_ = [], []
    for k in range(0, HORIZON + 1, 64):
        if k:
            c.run(64)
        wv, av = wet_counts(m, c.get_state()[0])
        wv_.append(wv)
        av_.append(av)
    c.close()
    out["n_wet"], out["n_act"] = float(np.mean(wv_)), float(np.mean(av_))
    return w, out


DENSE_LAYER = 1.0  # m of material added on every cell for the dense forward case


# the path's one-pass forward bytes per cell-update without the kept slopes (state in and out,
# static coefficients, material and level bytes, neighbour table)
ONE_PASS_BYTES = {"fp64": 124, "fp32": 72}
FWD_STEPS = 1000      # the forward-at-scale workload as specified: 1000 steps
DENSE_STEPS = 300     # the dense case that carries the step kernel's roofline


def forward_config2(args, ws, local):
    """Forward steps alone on the 3.75M-cell adaptive workload, through da_forward_run (the
    multi-step kernel), in both precisions: the workload as specified (three piles on a 20 km
    hill, FWD_STEPS steps: a sparse flow, tile culling skips the dry tiles; FP32-split's error
    against FP64 -- which equals the oracle bit for bit -- is reported after the last step) and a
    dense case on the same mesh with a layer of DENSE_LAYER m added on every cell, so that every
    cell is wet and updated every step.  The dense case carries the roofline of the step kernel;
    the launch shape of each run is the autotuner's."""
    from discrete_adjoint_b200 import GeoflowContext, TimeProps, _ffi, inputs
    w = inputs.workload2()
    m = w.mesh
    res = {}
    final = {}
    hbm, peak_kind = peaks()
    for name, prec, layer in (("fp32", _ffi.DA_PREC_FP32_SPLIT, 0.0),
                              ("fp32_dense", _ffi.DA_PREC_FP32_SPLIT, DENSE_LAYER),
                              ("fp64", _ffi.DA_PREC_FP64, 0.0),
                              ("fp64_dense", _ffi.DA_PREC_FP64, DENSE_LAYER)):
        steps = DENSE_STEPS if layer > 0 else FWD_STEPS
        c = GeoflowContext(w.mat, TimeProps(), precision=prec, device=local)
        c.upload_mesh(m)
        c.set_state(m.h0 + layer, m.hu0, m.hv0)
        tune = c.autotune(5)
        c.set_state(m.h0 + layer, m.hu0, m.hv0)
        c.set_time(0.0, 0)
        _, ms = c.run_timed(steps)
        ms = allmax(ms, ws, local)
        state = c.get_state()
        if layer == 0:
            final[name] = state
        wv, av = wet_counts(m, state[0])
        r = {"value": m.n * steps * ws / (ms * 1e-3), "steps": steps, "us_per_step": 1e3 * ms / steps,
             "wet_cells": wv, "active_cells": av,
             "launch_shape": {"blocks_per_sm": tune["best"][0], "grid": tune["best"][1]}}
        if layer > 0:
            pn = "fp64" if prec == _ffi.DA_PREC_FP64 else "fp32"
            bytes_step = algorithmic_bytes(pn, av)["k_steps"]
            gbs = bytes_step / (ms * 1e-3 / steps) / 1e9
            one_pass = ONE_PASS_BYTES[pn] * av / (ms * 1e-3 / steps) / 1e9
            r["roofline"] = {"kernel": "k_steps", "alg_bytes_per_step": bytes_step,
                             "bytes_per_cell_update": bytes_per_cell_update(pn)["forward"], "achieved": gbs,
                             "peak": hbm, "unit": "GB/s", "frac": gbs / hbm, "peak_kind": peak_kind,
                             "traffic": TRAFFIC_DENSE_PER_STEP[pn],
                             "frac_one_pass": one_pass / hbm, "one_pass_bytes_per_cell": ONE_PASS_BYTES[pn]}
        res[name] = r
        c.close()
    rl2 = lambda x, y: float(np.linalg.norm(x - y) / max(np.linalg.norm(y), 1e-300))  # noqa: E731
    a, b = final["fp64"], final["fp32"]
    err = {"h_rel_l2": rl2(b[0], a[0]), "hu_rel_l2": rl2(b[1], a[1]), "hv_rel_l2": rl2(b[2], a[2])}
    err["within_1e-5"] = max(err.values()) <= 1e-5
    res["fp32_rel_err_vs_fp64_after_%d_steps" % FWD_STEPS] = err
    return w, res


def ensemble_config4(args, ws, rank, local):
    """The batched ensemble: seeded members (plane slope U(20, 35) deg, pile volume U(1e4, 1e6) m^3,
    basal friction U(12, 28) deg, meshes of 16k-262k cells), forward + adjoint of each member's
    runout functional over 300 steps with 32 checkpoints, all members in the same launches; the
    same members run one after another through the plain FP64 single-instance path for the
    batched-vs-sequential ratio (device time of each run, summed).  With N ranks the members
    are split by a size-balanced greedy partition and each rank runs its share; the per-member
    results are gathered once."""
    from discrete_adjoint_b200 import Ensemble, GeoflowContext, Member, TimeProps, _ffi, adjoint_run, inputs
    from discrete_adjoint_b200.ensemble import gather_results, shard_members
    specs = inputs.ensemble_specs(args.members)
    sizes = [s.side * s.side for s in specs]
    mine = shard_members(sizes, ws, rank)
    members = []
    for k in mine:
        mesh, mat, _, box = inputs.ensemble_member(specs[k])
        members.append(Member(mesh, mat, box))
    cells = sum(mb.mesh.n for mb in members)
    total_cells = int(allsum(cells, ws, local))
    out = {"members": args.members, "cells": total_cells, "steps": ENS_STEPS, "snapshots": ENS_SNAPSHOTS,
           "members_per_rank_max": int(allmax(len(members), ws, local))}
    grads = {}
    for name, prec in (("fp64", _ffi.DA_PREC_FP64), ("fp32", _ffi.DA_PREC_FP32_SPLIT)):
        with Ensemble(members, precision=prec, device=local) as ens:
            tune = ens.autotune(5)
            ens.adjoint(ENS_STEPS, ENS_SNAPSHOTS)  # warm-up
            barrier(ws, local)
            g, ms = ens.adjoint(ENS_STEPS, ENS_SNAPSHOTS)
            barrier(ws, local)
            ms = allmax(ms, ws, local)
        grads[name] = gather_results({k: (gg.J, gg.dJ_dbedfrict[0], gg.dJ_dpile[0]) for k, gg in zip(mine, g)}, ws)
        out[name] = {"ms": ms, "value": total_cells * ENS_STEPS / (ms * 1e-3),
                     "launch_shape": {"blocks_per_sm": tune["best"][0], "grid": tune["best"][1]}}
    rel = lambda a, b: abs(a - b) / max(abs(b), 1e-300)  # noqa: E731
    out["fp32_rel_err_vs_fp64_max"] = {
        q: max(rel(grads["fp32"][k][i], grads["fp64"][k][i]) for k in grads["fp64"])
        for i, q in enumerate(("J", "dJ_dbedfrict", "dJ_dpile"))}
    # the FP32-split batched rate counts only with every member's J and gradients within 1e-4 of FP64
    fp32_ok = max(out["fp32_rel_err_vs_fp64_max"].values()) <= 1e-4
    out["fp32"]["within_tolerance"] = fp32_ok
    if not fp32_ok:
        out["fp32_out_of_tolerance"] = out.pop("fp32")
    if ws == 1 and not args.no_sequential:
        seq_ms, worst = 0.0, 0.0
        for i, mb in enumerate(members):
            with GeoflowContext(mb.mat, TimeProps(), precision=_ffi.DA_PREC_FP64, device=local) as c:
                c.upload_mesh(mb.mesh)
                c.set_state(mb.mesh.h0, mb.mesh.hu0, mb.mesh.hv0)
                if i == 0:
                    adjoint_run(c, mb.box, ENS_STEPS, ENS_SNAPSHOTS, mb.mesh.dh0_dpile[0])  # module warm-up
                gs = adjoint_run(c, mb.box, ENS_STEPS, ENS_SNAPSHOTS, mb.mesh.dh0_dpile[0])
            seq_ms += gs.device_ms
            e = grads["fp64"][mine[i]]
            worst = max(worst, rel(e[0], gs.J), rel(e[1], gs.dJ_dbedfrict[0]), rel(e[2], gs.dJ_dpile[0]))
        out["sequential_fp64"] = {"ms": seq_ms, "value": total_cells * ENS_STEPS / (seq_ms * 1e-3)}
        out["batched_fp64_over_sequential"] = seq_ms / out["fp64"]["ms"]
        if "fp32" in out:
            out["batched_fp32_over_sequential"] = seq_ms / out["fp32"]["ms"]
        out["batched_vs_sequential_max_rel_diff"] = worst
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3, help="timed forward+adjoint runs (512 time steps each)")
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=5)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-clocks", action="store_true")
    ap.add_argument("--no-forward", action="store_true", help="skip the forward-only section")
    ap.add_argument("--members", type=int, default=512, help="ensemble members (0 skips the ensemble section)")
    ap.add_argument("--no-sequential", action="store_true", help="skip the sequential baseline of the ensemble")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)

    ws, rank, local = dist_init(args.impl)
    if args.impl == "reference":
        # rank 0 alone runs the CPU reference; the other ranks exit without work (no process
        # group: nothing is exchanged)
        run_reference_arm(args, ws, rank)
        return

    from discrete_adjoint_b200 import inputs
    w, r = fwdadj(args, ws, local)
    m = w.mesh
    a, b = r["fp64"]["grad"], r["fp32"]["grad"]
    rel = lambda x, y: abs(x - y) / max(abs(y), 1e-300)  # noqa: E731
    rl2 = lambda x, y: float(np.linalg.norm(x - y) / max(np.linalg.norm(y), 1e-300))  # noqa: E731
    sa, sb = r["fp64"]["state"], r["fp32"]["state"]
    errs = {"h_rel_l2": rl2(sb[0], sa[0]), "hu_rel_l2": rl2(sb[1], sa[1]), "hv_rel_l2": rl2(sb[2], sa[2]),
            "J": rel(b.J, a.J), "dJ_dpile": rel(b.dJ_dpile[0], a.dJ_dpile[0]),
            "dJ_dbedfrict": rel(b.dJ_dbedfrict[0], a.dJ_dbedfrict[0]),
            "dJ_dintfrict": rel(b.dJ_dintfrict, a.dJ_dintfrict),
            "lambda0_rel_l2": rl2(b.lambda0, a.lambda0)}
    # the FP32-split run is the headline only within the stated tolerance: 1e-5 relative L2 on the
    # state, 1e-4 on every gradient; otherwise the plain FP64 path (bit-identical to the
    # reference's step()) is
    fp32_ok = (max(errs["h_rel_l2"], errs["hu_rel_l2"], errs["hv_rel_l2"]) <= 1e-5 and
               max(errs["dJ_dpile"], errs["dJ_dbedfrict"], errs["dJ_dintfrict"], errs["lambda0_rel_l2"]) <= 1e-4)
    head = "fp32" if fp32_ok and r["fp32"]["value"] > r["fp64"]["value"] else "fp64"
    hr = r[head]

    # roofline of the dominant kernel of the traced headline run
    tr = hr["trace"]
    dom = max(tr, key=lambda k: tr[k][0])
    alg = algorithmic_bytes(head, r["n_act"])
    hbm, peak_kind = peaks()
    avg_ms = tr[dom][0] / tr[dom][1]
    steps_per_launch = tr[dom][2] / tr[dom][1]
    achieved = alg.get(dom, 0.0) * steps_per_launch / (avg_ms * 1e-3) / 1e9

    fwd = None
    if not args.no_forward:
        w2, f2 = forward_config2(args, ws, local)
        fwd = {"workload": w2.name, "cells": w2.mesh.n, "unit": "cell-updates/s", **f2}

    ens = ensemble_config4(args, ws, rank, local) if args.members > 0 else None

    cpu = None
    if rank == 0 and ws == 1 and not args.no_cpu:
        rc = reference_fwdadj(2, 0)
        cpu = {"value": rc["value"], "unit": "cell-updates/s", "cores": rc["cores"], "kind": rc["kind"],
               "sample": rc["sample"]}

    if rank == 0:
        launches_per_run = sum(v[1] for v in tr.values())
        line = {
            "metric": METRIC, "value": hr["value"], "unit": "cell-updates/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": hr["ms"] / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64" if head == "fp64" else "f32", "data": "synthetic",
            "config": {"workload": HEADLINE_WORKLOAD, "cells": m.n, "horizon": HORIZON, "snapshots": SNAPSHOTS,
                       "functional": "sum h^2 dx dy over box " + str(inputs.WORKLOAD3_BOX),
                       "precision": "fp64" if head == "fp64" else "fp32-split",
                       "parallelism": f"replicas x{ws}" if ws > 1 else "single GPU",
                       "l2": "per-run working set larger than L2 (no flush needed)",
                       "forward_steps_per_run": hr["forward_steps"], "launch_shape": hr["launch_shape"]},
            "fp64": {"value": r["fp64"]["value"], "ms_per_run": r["fp64"]["ms"] / args.steps},
            "fp32_split": {"value": r["fp32"]["value"], "ms_per_run": r["fp32"]["ms"] / args.steps,
                           "over_fp64": r["fp32"]["value"] / r["fp64"]["value"], "rel_err_vs_fp64": errs,
                           "within_tolerance": fp32_ok, "e2e": r["fp32"]["e2e"]["value"]},
            "roofline": {"bound": "hbm", "kernel": dom, "achieved": achieved, "peak": hbm, "unit": "GB/s",
                         "frac": achieved / hbm, "peak_kind": peak_kind,
                         "alg_bytes_per_launch": alg.get(dom, 0.0) * steps_per_launch,
                         "bytes_per_cell_update": bytes_per_cell_update(head),
                         "alg_cells": "active cells (wet or next to a wet cell), the cells the kernel processes",
                         "steps_per_launch": steps_per_launch,
                         "avg_launch_ms": avg_ms, "wet_cells_avg": r["n_wet"], "active_cells_avg": r["n_act"],
                         "trace_ms_launches_steps": {k: [round(v[0], 4), v[1], v[2]] for k, v in tr.items()},
                         "traffic": traffic_per_launch(head, dom, r["n_act"], steps_per_launch),
                         "note": "the flow covers ~40 of 4096 tiles: the step is bound by the latency of its "
                                 "grid barriers and of one tile's dependent FP64 chain, not by HBM; the few "
                                 "active tiles stay in L2 between steps"},
            "e2e": hr["e2e"],
            "gpu_launches": int(launches_per_run * args.steps),
            "clocks": hr["clocks"],
            "cpu_baseline": cpu,
            "forward_only": fwd,
            "ensemble": ens,
        }
        print(json.dumps(line))
    if ws > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
