#!/usr/bin/env python
"""Benchmark of the headline workload: SU(3) Wilson HMC on a 32^4 lattice,
beta = 6.0, Omelyan (2mn) integrator with epsilon = 0.5 and 20 substeps
(tau = 1), mixed precision (FP32 links, momenta and force; FP64 action and
Hamiltonian sums, dH and Metropolis on the device), after thermalisation from
a hot start with seed 7. One step = one HMC trajectory; the metric is
trajectories per second.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Under torchrun (N > 1) every rank runs an independent replica chain on its own
GPU (the path has no exchange step: replicas only); value = total
trajectories of all ranks / max over ranks of the timed region.

--impl reference times the reference's algorithm on the host CPU cores: the
C++ restatement of src/gauge + src/lattice (oracle/, compiled with g++
-fopenmp), one momentum step + one link update + one plaquette of the same
32^4 FP32 fields per step, extrapolated to a trajectory.
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

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = dict(name="su3_hmc_32^4_beta6.0_2mn_eps0.5_n20_mixed", group=3, dims=[32, 32, 32, 32], beta=6.0,
                scheme="2mn", eps=0.5, substeps=20, seed=7, therm=200)
METRIC = "SU(3) 32^4 HMC trajectories/s"
UNIT = "traj/s"
# timed CPU work of the reference arm (complete trajectories, at least one)
REF_TIME_LIMIT = 120.0


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--therm", type=int, default=WORKLOAD["therm"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-physics", action="store_true",
                    help="skip the FP64-vs-mixed-precision chains of the headline line")
    ap.add_argument("--physics-traj", type=int, default=100,
                    help="trajectories of each chain of the FP64-vs-mixed comparison")
    ap.add_argument("--no-landau", action="store_true", help="skip the one-configuration Landau number")
    ap.add_argument("--lattice", type=int, default=32,
                    help="extent L of the L^4 lattice (32 = the headline workload; smaller for profiling captures)")
    ap.add_argument("--dims", type=int, nargs=4, default=None,
                    help="the four extents of a non-hypercubic lattice for profiling captures (overrides --lattice)")
    ap.add_argument("--workload", choices=["hmc", "batch", "landau", "wilson", "heatbath", "fp64-8x4"], default="hmc",
                    help="hmc: the headline line; batch: 64 SU(2) replicas in one persistent launch against 64 "
                         "separate chains; landau: time to theta < 1e-12, overrelaxation vs Fourier-accelerated "
                         "(plain and learned multiplier); wilson: all r x t Wilson loops of a thermalised "
                         "configuration; heatbath: heat-bath + overrelaxation sweeps; fp64-8x4: the FP64 8^4 "
                         "cold-start chain against the CPU oracle, trajectory by trajectory")
    ap.add_argument("--configs", type=int, default=2, help="landau workload: number of configurations")
    ap.add_argument("--fa-accept", choices=["theta", "functional"], default="functional",
                    help="landau workload: acceptance test of the Fourier-accelerated steps")
    ap.add_argument("--methods", default="or,plain,learned",
                    help="landau workload: solvers to run (or, plain, fixed, learned)")
    ap.add_argument("--fixed", default="0.08,0.6", help="landau workload: the fixed multiplier member alpha,high")
    ap.add_argument("--weights", default=None, help="landau workload: network file (default: the committed one)")
    ap.add_argument("--fp64", action="store_true",
                    help="hmc workload: the plain all-FP64 chain (links, momenta, force in FP64) instead of the "
                         "mixed-precision one, for the FP64-vs-mixed comparison")
    a = ap.parse_args()
    if a.dims:
        WORKLOAD["dims"] = list(a.dims)
        WORKLOAD["name"] = WORKLOAD["name"].replace("32^4", "x".join(map(str, a.dims)))
    elif a.lattice != 32:
        WORKLOAD["dims"] = [a.lattice] * 4
        WORKLOAD["name"] = WORKLOAD["name"].replace("32^4", f"{a.lattice}^4")
    if a.fp64:
        WORKLOAD["name"] = WORKLOAD["name"].replace("_mixed", "_fp64")
    WORKLOAD["prec_bytes"] = 8 if a.fp64 else 4
    return a


def sizes(dims, prec_bytes=4):
    V = 1
    for d in dims:
        V *= d
    nd = len(dims)
    U = nd * V * 18 * prec_bytes
    P = nd * V * 8 * prec_bytes
    return V, U, P


def deltas_counts(n):
    n_u = (n + 1) // 2
    return n_u, n - n_u


def algorithmic_bytes_per_traj(dims, n, prec_bytes=4):
    """Compulsory HBM bytes of one trajectory, every object read/written once:
    n_P (|U| + 2|P|) + n_U (2|U| + |P|) + |P| + 2(|U| + |P|) + 2|U|."""
    _, U, P = sizes(dims, prec_bytes)
    n_u, n_p = deltas_counts(n)
    return n_p * (U + 2 * P) + n_u * (2 * U + P) + P + 2 * (U + P) + 2 * U


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as fh:
            d = json.load(fh)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


KERNEL_DESC = {
    "line": "k_md_line<float,...,rows01,fused> (SU(3) line march: six plaquettes per site computed once, lower "
            "staples along x1 and x3 handed over, along x0 and x2 summed per link; momentum update and the "
            "following link update in the same pass)",
    "site": "k_momentum_step_site<SU3,float,4,..,rows01,fused> (staples + force + momentum update + the following "
            "link update, one thread per site; links read as rows 0,1, row 2 rebuilt)",
    "stored plaquettes": "k_md_plaquettes + k_md_transport<SU3,float,4,fused> (the projected plaquettes of every plane, "
                         "a warp per plane; the forces transported from them, momentum update and the following link "
                         "update, a warp per direction; times and traffic are the pair's)",
    "stored products": "k_md_products + k_md_force<double,4,fused> (the products of two links at a site, a warp per plane; "
                       "the forces from them and the following link update, a warp per direction; the pairs' time)",
    "separate": "momentum step and link update as two kernels",
}


def chosen_variant(report, prefix):
    """the launch variant the autotuner chose for the first key starting with
    `prefix` (e.g. 'line/128thr/4blk/f32x2'), or 'separate'"""
    for ln in report.splitlines():
        if ln.startswith(prefix) and "chosen " in ln:
            c = ln.split("chosen ", 1)[1].split(" [", 1)[0]
            return "separate" if c.startswith("separate") else c
    return "unknown"


def ncu_traffic(key):
    """DRAM bytes per launch of the dominant kernel from the data file of ncu
    captures (profiles/dram_traffic.json, keyed by the launch variant of the
    32^4 workload); null when the file has no entry"""
    p = os.path.join(ROOT, "profiles", "dram_traffic.json")
    try:
        with open(p) as fh:
            return float(json.load(fh)[key]["bytes_per_launch"])
    except (OSError, KeyError, ValueError, TypeError):
        return None


class Clocks:
    """nvidia-smi samples (every 200 ms) during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
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
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
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
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def cpu_trajectories(U_host, dims, deltas, beta, seed, count=1, time_limit=None, threads=0):
    """Complete trajectories of the reference algorithm (the oracle's C++
    restatement of runHmcUpdate, FP32, OpenMP on the host cores) on the full
    lattice: momentum refresh, H_old, the MD steps of `deltas`, reunitisation,
    H_new and the Metropolis test, timed one by one. Runs `count`
    trajectories, or stops early once `time_limit` seconds are spent (at
    least one). Returns (seconds per trajectory list, cores)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle

    pyoracle.build()
    cores = pyoracle.set_threads(threads)
    U = U_host
    times = []
    for k in range(count):
        t0 = time.perf_counter()
        U, _ = pyoracle.hmc_chain(WORKLOAD["group"], 1, dims, U, beta, deltas, seed, k, 1)
        times.append(time.perf_counter() - t0)
        if time_limit is not None and sum(times) >= time_limit:
            break
    return times, cores


def chain_stats(hist, bin_size=10):
    """plaquette mean with the standard error from bins of `bin_size`
    trajectories, acceptance, <exp(-dH)> with its binned error, mean dH"""
    import numpy as np

    def binned(x):
        x = np.asarray(x, dtype=np.float64)
        nb = len(x) // bin_size
        if nb < 2:
            return float(x.mean()), float("nan")
        b = x[:nb * bin_size].reshape(nb, bin_size).mean(axis=1)
        return float(x.mean()), float(b.std(ddof=1) / np.sqrt(nb))

    p, pe = binned(hist["plaq_history"])
    e, ee = binned(np.exp(-np.asarray(hist["deltaH_history"])))
    return {"trajectories": int(len(hist["plaq_history"])), "plaquette": p, "plaquette_err": pe,
            "acceptance": float(np.mean(hist["accept_history"])), "exp_minus_dH": e, "exp_minus_dH_err": ee,
            "dH_mean": float(np.mean(hist["deltaH_history"]))}


def physics_fp64_vs_mixed(ctx, U_host, grid, d, beta, ntraj):
    """Two chains from the same thermalised links and the same seed (so the
    same momentum and Metropolis streams): the mixed-precision one (FP32
    links, momenta, force; FP64 sums, dH, Metropolis) and the all-FP64 one,
    `ntraj` trajectories each. Errors from bins of 10 trajectories; the
    plaquette difference is compared with the two errors combined as if the
    chains were independent (they are correlated, so this is conservative)."""
    import numpy as np

    import mesh_gb300 as mg

    res = {}
    t = {}
    for name, prec, arr in (("mixed", mg.F32, U_host), ("fp64", mg.F64, U_host.astype(np.float64))):
        h = mg.Hmc(ctx, 3, prec, grid, seed=11)
        h.U.import_(arr)
        t0 = time.perf_counter()
        h.run(beta, d, ntraj, use_graph=True)
        h.history()
        t[name] = time.perf_counter() - t0
        res[name] = chain_stats(h.history())
        res[name]["traj_per_s"] = ntraj / t[name]
        h.close()
    dp = res["mixed"]["plaquette"] - res["fp64"]["plaquette"]
    err = float(np.hypot(res["mixed"]["plaquette_err"], res["fp64"]["plaquette_err"]))
    res["plaquette_diff"] = dp
    res["plaquette_diff_err"] = err
    res["within_2_sigma"] = bool(abs(dp) < 2 * err)
    res["run"] = (f"{ntraj} trajectories per chain from the headline chain's thermalised links, seed 11, "
                  f"2mn eps={WORKLOAD['eps']} n={WORKLOAD['substeps']}, beta={beta}")
    return res


def landau_one_config(ctx, L=24, therm=100):
    """Landau gauge fixing of one thermalised SU(3) L^4 beta = 6.0
    configuration (HMC seed 1, Haar-random transform seed 5) to
    theta < 1e-12: FP64 overrelaxation (omega 1.7), Fourier acceleration with
    the plain and with the learned multiplier (steps accepted on the gauge
    functional, overrelaxation fallback): seconds, iterations, fallbacks,
    functional."""
    from mesh_gb300 import landau_learn as ll

    (beta, Uh), = list(ll.hmc_configs(ctx, L, [6.0], [1], therm, 1, 0))
    params, _ = ll.load_weights()
    out = {"lattice": [L] * 4, "thermalisation": f"{therm} trajectories, seed 1", "transform_seed": 5}
    for method in ("or", "plain", "learned"):
        U = ll.prepared_links(ctx, Uh, transform_seed=5)
        r = ll.solve(ctx, U, method, params, beta)
        out[method] = {k: r[k] for k in ("seconds", "iterations", "fallbacks", "theta", "functional")}
        U.close()
    for m in ("plain", "learned"):
        out[f"speedup_{m}_vs_or"] = out["or"]["seconds"] / out[m]["seconds"]
    return out


# ---------------------------------------------------------------------------
def replica_seed(rank):
    """each rank's chain is an independent replica: its own seed"""
    return WORKLOAD["seed"] + rank


def job_time_and_rate(ms, steps, world, dist=None, device="cpu"):
    """(max over ranks of the timed region in ms, whole-job trajectories/s):
    every rank ran `steps` trajectories of its own replica, so the job did
    world x steps in the slowest rank's time"""
    if dist is not None:
        import torch

        t = torch.tensor([float(ms)], dtype=torch.float64, device=device)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    return ms, world * steps / (ms / 1000.0)


def run_reference(args):
    """The reference's algorithm on the host cores (the oracle restatement,
    FP32 = the reference's precision=1 path, all host threads): every step
    is one complete trajectory of the 32^4 workload. One untimed trajectory
    first; the timed steps stop after REF_TIME_LIMIT seconds (at least one),
    so that the run ends within a few minutes; `steps` reports how many ran."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    import numpy as np

    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle

    pyoracle.build()
    dims = WORKLOAD["dims"]
    d = pyoracle.make_deltas(WORKLOAD["scheme"], WORKLOAD["eps"], WORKLOAD["substeps"])
    U = pyoracle.random_gauge(3, 1, dims, WORKLOAD["seed"])
    warm, cores = cpu_trajectories(U, dims, d, WORKLOAD["beta"], WORKLOAD["seed"], count=min(1, args.warmup))
    times, cores = cpu_trajectories(U, dims, d, WORKLOAD["beta"], WORKLOAD["seed"] + 1, count=args.steps,
                                    time_limit=REF_TIME_LIMIT)
    value = len(times) / sum(times)
    sample = (f"{len(times)} complete trajectories ({WORKLOAD['scheme']} n={WORKLOAD['substeps']}: momentum "
              f"refresh, two actions, {len(d) // 2 + 1} link updates, {len(d) // 2} momentum steps, "
              f"reunitisation, Metropolis) of the reference algorithm on the full 32^4 SU(3) FP32 lattice, "
              f"{np.mean(times):.1f} s each, timed one by one after {len(warm)} untimed; capped at "
              f"{REF_TIME_LIMIT:.0f} s of timed work")
    line = {"metric": METRIC, "value": value, "unit": UNIT, "impl": "reference", "n_gpus": args.gpus,
            "steps": len(times), "warmup": len(warm), "ms_per_step": 1000.0 / value, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD["name"], "lattice": dims, "beta": WORKLOAD["beta"],
                       "integrator": f"{WORKLOAD['scheme']} eps={WORKLOAD['eps']} n={WORKLOAD['substeps']}",
                       "precision": "FP32 (the reference's precision=1 path)", "parallelism": "cpu threads",
                       "steps_requested": args.steps, "warmup_requested": args.warmup},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def run_ours(args):
    import numpy as np
    import torch

    import mesh_gb300 as mg

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import torch.distributed as dist

        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    mg.load()
    stream = torch.cuda.Stream()
    ctx = mg.Context(local, stream.cuda_stream)
    dims = WORKLOAD["dims"]
    grid = mg.Grid(dims)
    beta = WORKLOAD["beta"]
    d = mg.make_deltas(WORKLOAD["scheme"], WORKLOAD["eps"], WORKLOAD["substeps"])
    n = len(d)
    n_u, n_p = deltas_counts(n)
    pb = WORKLOAD["prec_bytes"]
    h = mg.Hmc(ctx, WORKLOAD["group"], mg.F64 if pb == 8 else mg.F32, grid, seed=replica_seed(rank))
    h.randomize_gauge_field()
    h.run(beta, d, args.therm, use_graph=True)
    # refresh, the first link update, n_p momentum steps each with the link update
    # after it (one launch fused, two from stored plaquettes or, in FP64, products:
    # at least, lattices beyond the scratch go in slabs), plaquette, metropolis,
    # accept copy
    stored = pb == 8 or chosen_variant(mg.tune_report(), "md_step/").startswith("stored")
    launches_per_traj = 1 + 1 + n_p * (2 if stored else 1) + 1 + 2
    h.run(beta, d, args.warmup, use_graph=True)
    ctx.synchronize()

    def barrier():
        if dist is not None:
            dist.barrier()

    clocks = Clocks(local)
    clocks.start()
    barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    h.run(beta, d, args.steps, use_graph=True)
    e1.record(stream)
    torch.cuda.synchronize()
    barrier()
    clk = clocks.stop()
    ms, value = job_time_and_rate(e0.elapsed_time(e1), args.steps, world, dist, device="cuda")
    hist = h.history(h.count - args.steps - args.warmup - args.therm)
    acc = float(np.mean(hist["accept_history"][-args.steps:]))
    plaq = float(np.mean(hist["plaq_history"][args.therm:]))
    edH = float(np.mean(np.exp(-hist["deltaH_history"][args.therm:])))

    # dominant kernel: the trajectory's fused MD step (staples + force + P
    # update + the link update after it, one thread per site), timed alone
    # with CUDA events on the launching stream; du = 0 leaves U unchanged.
    # Algorithmic bytes per launch: one momentum step (|U| + 2|P|) and one
    # link update (2|U| + |P|)
    _, Ub, Pb = sizes(dims, pb)
    B_f = Ub + 2 * Pb
    B_md = B_f + 2 * Ub + Pb
    U, P = h.U, h.P
    reps = 20
    for _ in range(3):
        h.md_step(beta, 1e-9, 0.0)
    torch.cuda.synchronize()
    f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    f0.record(stream)
    for _ in range(reps):
        h.md_step(beta, 1e-9, 0.0)
    f1.record(stream)
    torch.cuda.synchronize()
    t_md = f0.elapsed_time(f1) / reps / 1000.0
    for _ in range(3):
        h.momentum_step(beta, 1e-9)
    torch.cuda.synchronize()
    f0.record(stream)
    for _ in range(reps):
        h.momentum_step(beta, 1e-9)
    f1.record(stream)
    torch.cuda.synchronize()
    t_force = f0.elapsed_time(f1) / reps / 1000.0
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(stream)
    for _ in range(reps):
        mg.evolve(U, P, 0.0)
    ev1.record(stream)
    torch.cuda.synchronize()
    t_evolve = ev0.elapsed_time(ev1) / reps / 1000.0
    peak, peak_kind = measured_peaks()
    achieved = B_md / t_md / 1e9
    md_variant = "stored products" if pb == 8 else chosen_variant(mg.tune_report(), "md_step/")

    out = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak",
           "vs_baseline": None, "dtype": "f64" if pb == 8 else "f32", "data": "synthetic",
           "config": {"workload": WORKLOAD["name"], "lattice": dims, "beta": beta,
                      "integrator": f"{WORKLOAD['scheme']} eps={WORKLOAD['eps']} n={WORKLOAD['substeps']}",
                      "precision": "FP64 throughout" if pb == 8 else
                                   "FP32 links/momenta/force, FP64 sums/dH/Metropolis",
                      "thermalisation": f"{args.therm} trajectories from a hot start, seed {WORKLOAD['seed']}",
                      "parallelism": f"replicas x{world}" if world > 1 else "single GPU",
                      "l2": "inputs larger than L2 (links 302 MB + momenta 134 MB > 129 MB)",
                      "timing": "CUDA events on the launching stream, CUDA-graph replay of whole trajectories"},
           "physics": {"acceptance": acc, "plaquette_mean": plaq, "exp_minus_dH_mean": edH},
           "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                        "frac": achieved / peak,
                        "traffic": ncu_traffic(f"md_step/{md_variant}") if list(dims) == [32] * 4 else None,
                        "kernel": KERNEL_DESC.get(md_variant.split("/")[0], md_variant) + f" [{md_variant}]",
                        "algorithmic_bytes_per_launch": B_md, "avg_launch_ms": t_md * 1e3,
                        "peak_source": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured"
                        else "fallback 6.8 TB/s"},
           "kernels": {"momentum_step_alone_ms": t_force * 1e3,
                       "momentum_step_alone_GBps": B_f / t_force / 1e9,
                       "link_update_ms": t_evolve * 1e3,
                       "link_update_GBps": (2 * Ub + Pb) / t_evolve / 1e9,
                       "trajectory_algorithmic_GB": algorithmic_bytes_per_traj(dims, n, pb) / 1e9,
                       "trajectory_effective_GBps": algorithmic_bytes_per_traj(dims, n, pb) / (ms / args.steps / 1e3)
                       / 1e9},
           "clocks": clk, "gpu_launches": launches_per_traj * args.steps,
           "autotune": mg.tune_report().strip().splitlines()}

    # end to end through the C ABI with host buffers: the gauge field in the
    # reference's host layout is imported, one trajectory runs, the field is
    # exported back (pinned host memory), every step
    if not args.no_e2e:
        host_t = torch.empty((len(dims), grid.size, 18), dtype=torch.float64 if pb == 8 else torch.float32,
                             pin_memory=True)
        host = host_t.numpy()
        host[...] = U.export()
        k_e2e = max(3, min(args.steps, 10))
        h.run_host(host, beta, d, 1)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(k_e2e):
            h.run_host(host, beta, d, 1)
        t_e2e = (time.perf_counter() - t0) / k_e2e
        out["e2e"] = {"value": world / t_e2e, "unit": UNIT, "h2d_bytes_per_step": host.nbytes,
                      "d2h_bytes_per_step": host.nbytes + 40, "steps": k_e2e,
                      "api": "mesh_hmc_run_host (import U, one trajectory, export U)"}

    if rank == 0 and world == 1 and not args.no_cpu_baseline and pb == 4:
        times, cores = cpu_trajectories(U.export(), dims, list(d), beta, WORKLOAD["seed"] + 100, count=1)
        out["cpu_baseline"] = {"value": 1.0 / times[0], "unit": UNIT, "cores": cores, "kind": "port",
                               "sample": f"one complete trajectory ({times[0]:.1f} s: momentum refresh, two "
                                         f"actions, {n_u} link updates, {n_p} momentum steps, reunitisation, "
                                         f"Metropolis) of the reference algorithm (oracle/ C++ restatement, "
                                         f"FP32) on the full 32^4 lattice from this run's thermalised links"}
    if rank == 0 and world == 1 and not args.no_physics and pb == 4:
        out["physics_fp64_vs_mixed"] = physics_fp64_vs_mixed(ctx, U.export(), grid, d, beta, args.physics_traj)
    if rank == 0 and world == 1 and not args.no_landau and pb == 4:
        out["landau_24x4"] = landau_one_config(ctx)
    if rank == 0:
        print(json.dumps(out), flush=True)
    h.close()
    ctx.close()
    if dist is not None:
        dist.destroy_process_group()
    return 0


BATCH = dict(name="su2_batch_64rep_L{8,12,16,24}_beta[2.2,2.6]_2lf_eps0.5_n16_mixed", replicas=64,
             sizes=(8, 12, 16, 24), beta=(2.2, 2.6), seed=99, scheme="2lf", eps=0.5, substeps=16)


def batch_workload():
    """64 SU(2) replicas: extents uniform in {8,12,16,24}^4, beta uniform in
    [2.2, 2.6], drawn with seed 99; replica r uses seed r + 1"""
    import numpy as np

    rng = np.random.default_rng(BATCH["seed"])
    L = rng.choice(BATCH["sizes"], BATCH["replicas"])
    betas = rng.uniform(*BATCH["beta"], BATCH["replicas"])
    return [[int(x)] * 4 for x in L], betas, list(range(1, BATCH["replicas"] + 1))


def run_batch(args):
    """Batched replicas: aggregate link updates/s (sum over replicas of
    4 V_r x 16 MD steps per trajectory) for the whole batch in one persistent
    launch per trajectory step (CUDA-graph trajectory), against the same 64
    chains run one after the other (64 separate launch sequences)."""
    import numpy as np
    import torch

    import mesh_gb300 as mg

    torch.cuda.set_device(0)
    stream = torch.cuda.Stream()
    ctx = mg.Context(0, stream.cuda_stream)
    dims, betas, seeds = batch_workload()
    d = mg.make_deltas(BATCH["scheme"], BATCH["eps"], BATCH["substeps"])
    links = sum(4 * int(np.prod(x)) for x in dims)
    steps = args.steps
    therm = min(args.therm, 20)
    b = mg.HmcBatch(ctx, 2, mg.F32, dims, seeds)
    b.cold_start()
    b.run(betas, d, therm + args.warmup)

    def timed(fn):
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        fn()
        e1.record(stream)
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / 1000.0

    clocks = Clocks(0)
    clocks.start()
    t_batch = timed(lambda: b.run(betas, d, steps))
    clk = clocks.stop()
    acc = float(np.mean([b.history(r)["accept_history"][therm + args.warmup:].mean() for r in range(b.R)]))
    plaq = b.plaquettes()
    info = b.launch_info(len(d))
    md_launch = b.md_launch()
    chains = []
    for r in range(len(dims)):
        h = mg.Hmc(ctx, 2, mg.F32, mg.Grid(dims[r]), seed=seeds[r])
        h.cold_start()
        h.run(float(betas[r]), d, therm + args.warmup)
        chains.append(h)
    t_sep = timed(lambda: [h.run(float(betas[r]), d, steps) for r, h in enumerate(chains)])
    updates = links * BATCH["substeps"] * steps
    bytes_per_update = 84  # SU(2) FP32: force |U|+2|P| = 40 B, link update 2|U|+|P| = 44 B per link
    peak, _ = measured_peaks()
    out = {"metric": "SU(2) batched replicas link-updates/s", "value": updates / t_batch, "unit": "link-updates/s",
           "n_gpus": 1, "steps": steps, "warmup": args.warmup, "ms_per_step": t_batch / steps * 1e3,
           "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
           "config": {"workload": BATCH["name"], "replicas": len(dims), "links": links,
                      "sites": links // 4, "step": "one trajectory of every replica",
                      "start": f"cold, {therm} + {args.warmup} untimed trajectories",
                      "l2": f"inputs larger than L2 (links {links * 16 / 1e6:.0f} MB)"},
           "separate": {"value": updates / t_sep, "ms_per_step": t_sep / steps * 1e3,
                        "what": "the same 64 chains, each its own CUDA-graph trajectory, one after the other"},
           "speedup_vs_separate": t_sep / t_batch,
           "effective_GBps": updates * bytes_per_update / t_batch / 1e9, "peak_GBps": peak,
           "physics": {"acceptance": acc, "plaquette_mean": float(plaq.mean())},
           "gpu_launches": info["launches_per_trajectory"] * steps, "grids": info,
           "md_launch": md_launch, "clocks": clk}
    print(json.dumps(out), flush=True)
    return 0


def run_fp64_8x4(args):
    """SU(3) 8^4, beta = 5.7, FP64, cold start, 20 trajectories of 2lf
    epsilon = 0.5 n = 10 (tau = 1), momenta from seed 1234: plaquette, dH
    and accept per trajectory on the GPU chain and on the CPU oracle's chain
    (same counter-based streams), with trajectories per second of both."""
    import numpy as np
    import torch

    import mesh_gb300 as mg

    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle

    pyoracle.build()
    dims, beta, seed, ntraj = [8, 8, 8, 8], 5.7, 1234, 20
    d = mg.make_deltas("2lf", 0.5, 10)
    ctx = mg.Context(0)
    h = mg.Hmc(ctx, 3, mg.F64, mg.Grid(dims), seed=seed)
    h.cold_start()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    recs = [h.update(beta, d) for _ in range(ntraj)]
    t_gpu = time.perf_counter() - t0
    t0 = time.perf_counter()
    _, ro = pyoracle.hmc_chain(3, 2, dims, pyoracle.unit_gauge(3, 2, dims), beta, pyoracle.make_deltas("2lf", 0.5, 10),
                               seed, 0, ntraj)
    t_cpu = time.perf_counter() - t0
    rows = [{"traj": k, "plaq_gpu": r["plaquette"], "plaq_oracle": float(ro[k, 0]), "dH_gpu": r["dH"],
             "dH_oracle": float(ro[k, 1]), "accept_gpu": r["accept"], "accept_oracle": float(ro[k, 2])}
            for k, r in enumerate(recs)]
    out = {"metric": "SU(3) 8^4 FP64 HMC trajectories/s (cold start, per-trajectory parity)", "value": ntraj / t_gpu,
           "unit": "traj/s", "n_gpus": 1, "steps": ntraj, "higher_is_better": True, "dtype": "f64",
           "data": "synthetic", "config": {"workload": "su3_hmc_8^4_beta5.7_2lf_eps0.5_n10_fp64_cold_seed1234"},
           "cpu_oracle_traj_per_s": ntraj / t_cpu, "cpu_cores": pyoracle.set_threads(0),
           "max_abs_diff": {"plaquette": max(abs(r["plaq_gpu"] - r["plaq_oracle"]) for r in rows),
                            "dH": max(abs(r["dH_gpu"] - r["dH_oracle"]) for r in rows)},
           "accept_agree": all(r["accept_gpu"] == r["accept_oracle"] for r in rows), "rows": rows}
    print(json.dumps(out), flush=True)
    return 0


def run_heatbath(args):
    """Heat-bath + overrelaxation updates of SU(3) L^4 at beta = 6.0 in FP32
    (one heat-bath and three overrelaxation sweeps per step, from a cold start
    after `therm` such steps): link updates per second, and the bytes every
    link update must move (the link read and written, 2 x 72 B; the staple's
    neighbour links come from the caches) per second."""
    import torch

    import mesh_gb300 as mg

    torch.cuda.set_device(0)
    stream = torch.cuda.Stream()
    ctx = mg.Context(0, stream.cuda_stream)
    L = args.lattice
    U = mg.GaugeField(ctx, 3, mg.F32, mg.Grid([L] * 4)).set_unit()
    n_or = 3

    def step(k):
        mg.heatbath_sweep(U, 6.0, 7, k)
        for _ in range(n_or):
            mg.overrelax_sweep(U)

    therm = min(args.therm, 50)
    for k in range(therm + args.warmup):
        step(k)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for k in range(args.steps):
        step(therm + args.warmup + k)
    e1.record(stream)
    torch.cuda.synchronize()
    dt = e0.elapsed_time(e1) / 1000.0 / args.steps
    links = 4 * L ** 4
    upd = links * (1 + n_or) / dt
    peak, _ = measured_peaks()
    out = {"metric": "SU(3) heat-bath + overrelaxation link updates/s", "value": upd, "unit": "link-updates/s",
           "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
           "higher_is_better": True, "dtype": "f32", "data": "synthetic",
           "config": {"workload": f"su3_heatbath_{L}^4_beta6.0_1hb_{n_or}or", "start": f"cold, {therm} steps"},
           "effective_GBps": upd * 144 / 1e9, "peak_GBps": peak, "plaquette": mg.plaquette(U),
           "gpu_launches": 8 * (1 + n_or) * args.steps}
    print(json.dumps(out), flush=True)
    return 0


def run_wilson(args):
    """All rectangular Wilson loops W(r, t), r = 1..L/2, t = 1..L, of a
    thermalised SU(3) L^4 beta = 6.0 configuration (mixed-precision HMC,
    hot start, seed 7), FP32 links: loop sets per second and the effective
    bandwidth (every line extension reads two link objects and writes one per
    site, every loop sum reads the three spatial lines and the temporal line:
    four per site)."""
    import numpy as np
    import torch

    import mesh_gb300 as mg

    torch.cuda.set_device(0)
    ctx = mg.Context(0)
    L = args.lattice
    h = mg.Hmc(ctx, 3, mg.F32, mg.Grid([L] * 4), seed=7)
    h.randomize_gauge_field()
    h.run(6.0, mg.make_deltas("2mn", 0.5, 20), args.therm, use_graph=True)
    R, T = L // 2, L
    W = mg.wilson_loops(h.U, R, T)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        W = mg.wilson_loops(h.U, R, T)
    dt = (time.perf_counter() - t0) / args.steps
    V = L ** 4
    set_bytes = 72 * V * (3 * ((T - 1) + 3 * (R - 1)) + 4 * R * T)
    out = {"metric": "SU(3) Wilson loop sets/s", "value": 1.0 / dt, "unit": "sets/s", "n_gpus": 1,
           "steps": args.steps, "higher_is_better": True, "dtype": "f32", "data": "synthetic",
           "config": {"workload": f"su3_wilson_loops_{L}^4_r1..{R}_t1..{T}", "thermalisation": f"{args.therm} "
                      "trajectories, seed 7", "launches_per_set": (T - 1) + 3 * (R - 1) + R * T},
           "seconds_per_set": dt, "effective_GBps": set_bytes / dt / 1e9,
           "W": {f"{r + 1}x{t + 1}": float(W[r, t]) for r in range(min(R, 4)) for t in range(min(T, 4))}}
    print(json.dumps(out), flush=True)
    return 0


def run_landau(args):
    """Time to theta < 1e-12 from a Haar-random gauge transform of thermalised
    SU(3) L^4 beta = 6.0 configurations: FP64 overrelaxation (omega 1.7) and
    Fourier-accelerated steepest descent with the plain and the learned
    spectral multiplier (overrelaxation fallback)."""
    import numpy as np

    import mesh_gb300 as mg
    from mesh_gb300 import landau_learn as ll

    ctx = mg.Context(0)
    L = args.lattice
    seeds = np.arange(1, args.configs + 1)
    cfgs = ll.hmc_configs(ctx, L, [6.0] * len(seeds), seeds, args.therm, 1, 0)
    params, _ = ll.load_weights(args.weights) if args.weights else ll.load_weights()
    fixed = tuple(float(x) for x in args.fixed.split(","))
    methods = [m for m in args.methods.split(",") if m]
    rows = []
    for k, (beta, Uh) in enumerate(cfgs):
        for method in methods:
            U = ll.prepared_links(ctx, Uh, transform_seed=5)
            r = ll.solve(ctx, U, method, params, beta, accept=args.fa_accept, member=fixed)
            r["config"] = k
            r["seed"] = int(seeds[k])
            r["cost"] = r["iterations"] + 11 * r["fallbacks"]
            rows.append(r)
            print(json.dumps({"row": r}), flush=True)
            U.close()
    summ = {m: {"mean_seconds": float(np.mean([r["seconds"] for r in rows if r["method"] == m])),
                "mean_iterations": float(np.mean([r["iterations"] for r in rows if r["method"] == m])),
                "fallbacks": int(sum(r["fallbacks"] for r in rows if r["method"] == m)),
                "cost": int(sum(r["cost"] for r in rows if r["method"] == m))}
            for m in methods}
    lv = summ.get("learned", {}).get("mean_seconds")
    value = lv if lv is not None else summ[methods[0]]["mean_seconds"]
    out = {"metric": "Landau gauge fixing seconds to theta<1e-12", "value": value,
           "unit": "s", "n_gpus": 1, "steps": len(seeds), "higher_is_better": False, "dtype": "f64",
           "data": "synthetic", "config": {"workload": f"su3_landau_{L}^4_beta6.0_or1.7_vs_fa", "lattice": [L] * 4,
                                           "thermalisation": f"{args.therm} trajectories, seeds 1..{len(seeds)}",
                                           "transform": "Haar-random, seed 5", "fa_accept": args.fa_accept,
                                           "cost": "descent steps + 11 per overrelaxation fallback"},
           "summary": summ, "rows": rows, "fixed_member": fixed}
    if "or" in summ:
        for m in ("learned", "plain", "fixed"):
            if m in summ:
                out[f"speedup_{m}_vs_or"] = summ["or"]["mean_seconds"] / summ[m]["mean_seconds"]
    print(json.dumps(out), flush=True)
    return 0


def main():
    args = parse()
    if args.impl == "reference":
        return run_reference(args)
    if args.workload == "batch":
        return run_batch(args)
    if args.workload == "landau":
        return run_landau(args)
    if args.workload == "wilson":
        return run_wilson(args)
    if args.workload == "heatbath":
        return run_heatbath(args)
    if args.workload == "fp64-8x4":
        return run_fp64_8x4(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
