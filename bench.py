"""Benchmark: atom-evaluations/s of MOIL's nonbonded energy/force path on one GB300.

Workload (default): 512 independent periodic TIP3P boxes of uneven size (atom counts
log-uniform in [1500, 12000], whole molecules, 0.997 g/cm^3, rc 9 Å, alpha 0.35,
PME grid the smallest 2/3/5-smooth n >= 1 point/Å, order 4) evaluated together in one
batched, mixed-precision pass -- the path-image / milestoning-swarm shape.  A step is
one full nonbonded evaluation of every replica (real space + exclusion corrections +
PME + self), with the pair lists rebuilt every 10 steps as MOIL's '#lis 10' does.

    python bench.py [--steps K] [--warmup W] [--impl ours|reference] [--gpus N]

value      : atom-evals/s, coordinates and gradients resident in device memory
e2e        : the same through moil_nb_eval with pinned host buffers (copies timed)
roofline   : the dominant kernel against the FP32 pipe (pair math is FP32-bound)
cpu_baseline: the oracle (a C restatement of MOIL's FP64 routines, MOIL's own list path
             and erfc table) on a bounded sample of replicas, one host thread
plain_fp64 : the plain FP64 GPU path, one replica per launch, on a sample of replicas
pressure_analysis: MOIL's pressure-analysis terms (molecular virial tensor, moil_nb_pressure) of
             the whole batch, host buffers, wall clock per call (one evaluation + the pass)
single_system_md: one 96,000-atom water box through a 1,000-step rigid-water trajectory on the
             device (lists every 10 steps, 1.5 Å skin), whole steps timed, the FP64 path beside it
adjoint_64 : dE/dq, dE/deps, dE/dsigma per atom (moil_nb_adjoint) for 64 perturbed copies of the
             23,558-atom solute system in one batch, wall clock per call, the evaluation beside it
"""
from __future__ import annotations

import argparse
import json
import os
import platform
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "atom-evals/s mixed+batched vs plain FP64 on 1 GB300 at ≤1e-5 rel RMS force err"
F_PAIR = 50            # FP32 operations per in-cutoff site pair (FMA = 2, MUFU = 1)
LIST_PERIOD = 10
SKIN = 1.0
# DRAM bytes per water molecule of one water-kernel launch (ncu dram__bytes_read.sum +
# dram__bytes_write.sum): full lists (an earlier build, 74,171 waters) 37.44 MB, k_water_h (half
# lists, 256-water blocks, 48 replicas of 500-4,000 waters, 82,496 waters) 38.79 MB
WATER_KERNEL_DRAM_BYTES_PER_WATER = {1: 504.9, 2: 470.2}
WATER_KERNEL_NAME = {1: "k_water_s (full lists)", 2: "k_water_h (half lists)"}
# DRAM bytes per atom of one evaluation's PME kernels (k_pme_sites, k_plane_fwd, k_zconv_f,
# k_plane_inv, k_pme_gather_f: 5.96 + 4.42 + 12.05 + 12.02 + 16.59 MB, the same capture, 247,488
# atoms, caches flushed before each launch, so an upper bound)
PME_DRAM_BYTES_PER_ATOM = 206.3


ACCEL = 418.4                 # (kcal/mol/Å) / amu in Å/ps^2
KB = 0.0019872041             # kcal/mol/K


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def host_cpu():
    """The host's CPU model and logical core count (lscpu, else /proc/cpuinfo)."""
    model = None
    try:
        out = subprocess.run(["lscpu"], capture_output=True, text=True, timeout=10).stdout
        for line in out.splitlines():
            if line.split(":")[0].strip() == "Model name":
                model = line.split(":", 1)[1].strip()
                break
    except Exception:
        pass
    if not model:
        try:
            with open("/proc/cpuinfo") as f:
                for line in f:
                    if line.lower().startswith(("model name", "cpu model")):
                        model = line.split(":", 1)[1].strip()
                        break
        except Exception:
            pass
    return {"cpu_model": model or platform.processor() or platform.machine(), "nproc": os.cpu_count(),
            "arch": platform.machine()}


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f)
    except Exception:
        return {}


def fp32_peak_tflops(sm_mhz):
    """FP32 FMA peak of a 152-SM GB300 (128 FP32 lanes/SM, 2 flops per FMA) at sm_mhz."""
    return 152 * 128 * 2 * sm_mhz * 1e6 / 1e12


class ClockSampler:
    """Samples nvidia-smi clocks and throttle reasons while the timed region runs."""

    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index=0):
        self.index = index
        self.rows = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
            # nvidia-smi takes a moment to start: wait (at most 2 s) for its first row, then
            # keep only the rows that arrive inside the timed region
            t0 = time.perf_counter()
            while not self.rows and time.perf_counter() - t0 < 2.0:
                time.sleep(0.01)
            self.rows.clear()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def stop(self):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
            self.t.join(timeout=2)
        sm = []
        mx = 0.0
        reasons = set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in self.rows:
            try:
                sm.append(float(r[0]))
                mx = max(mx, float(r[1]))
                for k, nm in enumerate(names):
                    if r[4 + k].lower().startswith("active"):
                        reasons.add(nm)
            except Exception:
                continue
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx or None,
                "reasons": sorted(reasons), "samples": len(sm)}


def job_rate(units_local: float, seconds_local: float):
    """Whole-job throughput over the ranks of the default process group: the units every rank
    processed, summed, over the slowest rank's time (each rank times its own GPU).  Returns
    (units / s, slowest rank's seconds); a single process gives units / seconds."""
    import torch
    import torch.distributed as dist
    if not (dist.is_available() and dist.is_initialized()) or dist.get_world_size() == 1:
        return units_local / seconds_local, seconds_local
    u = torch.tensor([float(units_local)], dtype=torch.float64)
    t = torch.tensor([float(seconds_local)], dtype=torch.float64)
    dist.all_reduce(u, op=dist.ReduceOp.SUM)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(u[0]) / float(t[0]), float(t[0])


def build_workload(rank=0, n_rep=512):
    """The 512-replica batch; a smaller n_rep keeps the first n_rep replicas (profiling)."""
    from moil_fnrfd_gb300 import systems
    reps = systems.config3(512, seed=3000 + 7919 * rank)
    return reps[:n_rep]


def cpu_baseline(reps, budget_s=12.0):
    """The oracle, MOIL's list path + erfc table, one host thread, lists every 10 evals."""
    from oracle import oracle
    done_atoms = 0
    t0 = time.perf_counter()
    n = 0
    for s in reps:
        oracle.eforce_batch([s], mode="moil", nthreads=1, nevals=LIST_PERIOD, list_period=LIST_PERIOD)
        done_atoms += s.npt * LIST_PERIOD
        n += 1
        if time.perf_counter() - t0 > budget_s:
            break
    dt = time.perf_counter() - t0
    return {"value": done_atoms / dt, "unit": "atom-evals/s", "cores": 1, "kind": "port",
            "sample": f"{n} of {len(reps)} replicas x {LIST_PERIOD} evaluations (lists rebuilt once), "
                      f"oracle in MOIL list-path mode (13 image translations, erfc spline table, +2 Å buffers), "
                      f"{dt:.1f} s",
            "note": "one host thread, as MOIL runs one serial process per system", **host_cpu()}


def rigid_water_velocities(s, temperature, seed):
    """Maxwell-Boltzmann velocities (Å/ps) of an all-water system with each molecule's three
    bond-length rates removed (the velocity half of RATTLE): v_a += sum_k lambda_k d_k / m_a over
    the O-H1, O-H2 and H1-H2 constraints d_k = x_a - x_b, lambda from the 3x3 system per water
    that zeroes every d_k . (v_a - v_b)."""
    from moil_fnrfd_gb300.systems import MASS_H, MASS_O
    rng = np.random.Generator(np.random.PCG64(seed))
    m = np.tile([MASS_O, MASS_H, MASS_H], s.npt // 3).reshape(-1, 3)
    v = (rng.normal(size=(s.npt, 3)) * np.sqrt(KB * temperature * ACCEL / m.reshape(-1))[:, None]).reshape(-1, 3, 3)
    x = s.coor.reshape(-1, 3, 3)
    pairs = ((0, 1), (0, 2), (1, 2))
    d = np.stack([x[:, a] - x[:, b] for a, b in pairs], axis=1)
    M = np.empty((x.shape[0], 3, 3))
    for k, (a, b) in enumerate(pairs):
        for l, (c, e) in enumerate(pairs):
            coef = ((a == c) - (a == e)) / m[:, a] - ((b == c) - (b == e)) / m[:, b]
            M[:, k, l] = (d[:, k] * d[:, l]).sum(-1) * coef
    rhs = -np.stack([(d[:, k] * (v[:, a] - v[:, b])).sum(-1) for k, (a, b) in enumerate(pairs)], axis=1)
    lam = np.linalg.solve(M, rhs[..., None])[..., 0]
    for k, (a, b) in enumerate(pairs):
        v[:, a] += lam[:, k, None] * d[:, k] / m[:, a, None]
        v[:, b] -= lam[:, k, None] * d[:, k] / m[:, b, None]
    return v.reshape(-1, 3), m.reshape(-1)


def press_leg(nb, reps, coor, e2e_ms, calls=3):
    """moil_nb_pressure on the whole batch (every replica a TIP3P box, one molecule per water):
    one evaluation plus the molecular-virial pass per call, pinned host coordinates, energies
    and the twelve terms back (no gradient copy: the analysis reads the tensor), wall clock."""
    from moil_fnrfd_gb300.systems import MASS_H, MASS_O
    mol = np.concatenate([np.arange(s.npt, dtype=np.int32) // 3 for s in reps])
    mass = np.tile(np.array([MASS_O, MASS_H, MASS_H]), len(mol) // 3)
    nb.set_molecules(mol, mass)
    nb.pressure(coor, with_gradient=False)   # first call allocates the pass's buffers
    t = []
    for _ in range(calls):
        t0 = time.perf_counter()
        nb.pressure(coor, with_gradient=False)
        t.append((time.perf_counter() - t0) * 1e3)
    nb.set_molecules(None, None)
    ms = statistics.median(t)
    return {"ms_per_call": ms, "eval_e2e_ms": statistics.median(e2e_ms), "pass_ms": ms - statistics.median(e2e_ms),
            "calls": calls, "sample": "the timed batch, molecules = waters, no gradient copy"}


def adjoint_leg(local, calls=5):
    """Parameter derivatives (moil_nb_adjoint) of the sensitivity workload: 64 seeded +-1%
    perturbed copies of the 23,558-atom solute system in one batch.  One call is an evaluation
    (lists, positions, the PME grid recomputed) plus the adjoint kernels, pinned host
    coordinates in and the three per-atom derivative arrays out, wall clock (median of
    `calls`); moil_nb_eval of the same batch and buffers beside it."""
    import torch
    from moil_fnrfd_gb300 import systems as S
    from moil_fnrfd_gb300.nb import Nonbonded
    t0 = time.perf_counter()
    copies = S.perturbed_copies(S.config1(), 64)
    nb = Nonbonded(copies, device=local, skin=SKIN, list_period=LIST_PERIOD)
    natoms = sum(s.npt for s in copies)
    log(f"adjoint workload: {len(copies)} copies, {natoms} atoms, set up in {time.perf_counter() - t0:.1f} s")
    hc = torch.from_numpy(np.ascontiguousarray(np.concatenate([s.coor for s in copies]))).pin_memory().numpy()
    hd = torch.empty((natoms, 3), dtype=torch.float64).pin_memory().numpy()
    outs = [torch.empty(natoms, dtype=torch.float64).pin_memory().numpy() for _ in range(3)]

    def timed(fn):
        for _ in range(2):
            fn()
        t = []
        for _ in range(calls):
            t1 = time.perf_counter()
            fn()
            t.append((time.perf_counter() - t1) * 1e3)
        return statistics.median(t)

    adj_ms = timed(lambda: nb.adjoint_into(hc, *outs))
    eval_ms = timed(lambda: nb.eforce_into(hc, hd, want_energies=False))
    groups = nb.groups()
    nb.close()
    return {"workload": f"{len(copies)} perturbed copies (eps, sigma per LJ type and solute charges, +-1%) "
                        f"of the {copies[0].npt}-atom solute system, {natoms} atoms",
            "value": natoms / (adj_ms / 1e3), "unit": "atom-evals/s (dE/dq, dE/deps, dE/dsigma per atom)",
            "ms_per_call": adj_ms, "eval_ms": eval_ms, "cost_vs_eval": adj_ms / eval_ms, "calls": calls,
            "replica_groups": groups,
            "timing": "wall clock per call, pinned host buffers: H2D coordinates, D2H three derivative arrays"}


def accuracy_leg(nb, reps, d_coor, d_dpot, n_sample=6):
    """One batched evaluation of the timed coordinates; for n_sample replicas spread over the
    batch, each energy term's error relative to the term, |dE_total| / |E_total| and the
    relative RMS gradient error against the oracle (parity mode: MOIL's predicate, FP64)."""
    from oracle import oracle
    energies = nb.eforce_device(d_coor.data_ptr(), d_dpot.data_ptr())
    dp = d_dpot.cpu().numpy()
    offs = np.cumsum([0] + [s.npt for s in reps])
    terms = ("e_vdw", "e_el", "e_vsym", "e_lsym", "e_corr", "e_self", "e_ew_receip")
    picks = sorted(set(int(round(k * (len(reps) - 1) / max(n_sample - 1, 1))) for k in range(n_sample)))
    rows, worst = [], {k: 0.0 for k in terms}
    for r in picks:
        s = reps[r]
        ref, eref = oracle.eforce(s, mode="parity")
        e = energies[r]
        rel = {k: abs(e[k] - eref[k]) / abs(eref[k]) for k in terms if eref[k] != 0}
        for k, v in rel.items():
            worst[k] = max(worst[k], v)
        g = dp[offs[r]:offs[r + 1]]
        rows.append({"replica": r, "atoms": s.npt, "e_total": eref["e_total"],
                     "total_rel": abs(e["e_total"] - eref["e_total"]) / abs(eref["e_total"]),
                     "force_rel_rms": float(np.sqrt(((g - ref) ** 2).sum() / (ref ** 2).sum())),
                     "term_rel": {k: float(f"{v:.3g}") for k, v in rel.items()}})
    return {"oracle": "parity mode (MOIL's predicate at these coordinates, FP64)",
            "max_total_rel": max(x["total_rel"] for x in rows),
            "max_force_rel_rms": max(x["force_rel_rms"] for x in rows),
            "max_term_rel": {k: float(f"{v:.3g}") for k, v in worst.items()},
            "tolerance": {"total_rel": 1e-6, "force_rel_rms": 1e-5}, "replicas": rows}


def md_leg(local, steps=1000, warmup=20):
    """One 96,000-atom water box (32,000 TIP3P, 98.6 Å, rc 10, alpha 0.32, grid 100^3) through
    a rigid-water leapfrog trajectory on the device (moil_nb_md_step: evaluation, leapfrog and
    SETTLE each step, nothing copied to the host): 2 fs steps from 300 K, pair lists rebuilt
    every 10 steps with a 1.5 Å skin.  Timed by wall clock around the whole trajectory."""
    import torch
    from moil_fnrfd_gb300 import systems
    from moil_fnrfd_gb300.nb import MOIL_NB_FP64, Nonbonded
    s = systems.config2()
    nb = Nonbonded(s, device=local, skin=1.5, list_period=10)
    v0, m0 = rigid_water_velocities(s, 300.0, seed=11)
    x = torch.tensor(s.coor, dtype=torch.float64, device=f"cuda:{local}")
    v = torch.tensor(v0, dtype=torch.float64, device=x.device)
    m = torch.tensor(m0, dtype=torch.float64, device=x.device)
    torch.cuda.synchronize()
    nb.md_step(x.data_ptr(), v.data_ptr(), m.data_ptr(), 0.002, warmup)
    e, ek = nb.md_step(x.data_ptr(), v.data_ptr(), m.data_ptr(), 0.002, 1)
    e0 = e[0]["e_total"] + ek
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e, ek = nb.md_step(x.data_ptr(), v.data_ptr(), m.data_ptr(), 0.002, steps)
    torch.cuda.synchronize()
    wall = time.perf_counter() - t0
    e1 = e[0]["e_total"] + ek
    a, b, c = (x[k::3] for k in range(3))
    cerr = float((torch.linalg.vector_norm(b - a, dim=1) - systems.TIP3_ROH).abs().max())
    out = {"workload": "32,000 TIP3P waters (96,000 atoms), 98.6 Å box, rc 10 Å, alpha 0.32, PME 100^3, "
                       "rigid-water leapfrog (SETTLE) at 2 fs from 300 K on the device, lists every 10 steps, "
                       "1.5 Å skin",
           "steps": steps, "value": s.npt * steps / wall, "unit": "atom-evals/s (whole MD steps)",
           "ms_per_step": 1e3 * wall / steps, "ns_per_day": steps * 0.002e-3 / wall * 86400.0,
           "energy_total_start_end": [e0, e1], "constraint_err_A": cerr}
    nb.close()
    p = Nonbonded(s, precision=MOIL_NB_FP64, device=local)
    dc = torch.from_numpy(s.coor).to(f"cuda:{local}")
    dd = torch.empty_like(dc)
    p.eforce_device(dc.data_ptr(), dd.data_ptr())
    stp = torch.cuda.ExternalStream(p.stream())
    ta = torch.cuda.Event(enable_timing=True)
    tb = torch.cuda.Event(enable_timing=True)
    ta.record(stp)
    for _ in range(3):
        p.eforce_device(dc.data_ptr(), dd.data_ptr())
    tb.record(stp)
    torch.cuda.synchronize()
    out["plain_fp64_ms_per_eval"] = ta.elapsed_time(tb) / 3
    out["plain_fp64_atom_evals_per_s"] = s.npt / (out["plain_fp64_ms_per_eval"] / 1e3)
    p.close()
    return out


def run_reference(args):
    """Reference arm: MOIL's algorithm (the oracle restatement; MOIL's Fortran cannot be
    built here) on all host cores, same workload, metric and units."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from oracle import oracle
    reps = build_workload()
    threads = os.cpu_count() or 1
    sample = reps[:max(threads, 1) * 2]
    atoms = sum(s.npt for s in sample) * LIST_PERIOD
    times = []
    for it in range(args.warmup + args.steps):
        t0 = time.perf_counter()
        oracle.eforce_batch(sample, mode="moil", nthreads=threads, nevals=LIST_PERIOD, list_period=LIST_PERIOD)
        dt = time.perf_counter() - t0
        if it >= args.warmup:
            times.append(dt)
    value = atoms * len(times) / sum(times)
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "atom-evals/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * sum(times) / len(times),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic",
            "config": {"workload": "512 batched uneven TIP3P boxes (1500-12000 atoms each), rc 9, alpha 0.35",
                       "sample_per_step": f"{len(sample)} replicas x {LIST_PERIOD} evaluations"},
            "cpu_baseline": {"value": value, "unit": "atom-evals/s", "cores": threads, "kind": "port",
                             "sample": f"{len(sample)} of {len(reps)} replicas x {LIST_PERIOD} evaluations per step, "
                                       "OpenMP over replicas, oracle in MOIL list-path mode",
                             "label": "not MOIL: the oracle's all-core OpenMP variant (MOIL itself runs one "
                                      "serial process per system)", **host_cpu()},
            "e2e": {"value": value, "unit": "atom-evals/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    # 200 steps (about 0.5 s timed) give the 200 ms clock sampler a few samples under load
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--no-fp64", action="store_true", help="skip the plain FP64 leg")
    ap.add_argument("--replicas", type=int, default=512, help="first R replicas only (profiling captures)")
    ap.add_argument("--no-md", action="store_true", help="skip the single-system trajectory leg")
    ap.add_argument("--no-press", action="store_true", help="skip the pressure-analysis leg")
    ap.add_argument("--groups", type=int, default=0,
                    help="replica groups evaluated concurrently (0: the library's automatic choice)")
    ap.add_argument("--water-kernel", default="auto", choices=["auto", "full", "half"],
                    help="water-water kernel shape (moil_nb_set_shape; auto: the library's choice)")
    ap.add_argument("--half-block", type=int, default=0, choices=[0, 128, 256, 512],
                    help="waters per block of the half-list water kernel (0: the library's default)")
    ap.add_argument("--no-adj", action="store_true", help="skip the parameter-derivative (adjoint) leg")
    ap.add_argument("--no-tune", action="store_true",
                    help="skip the autotuner (it runs unless a shape is forced by --groups/--water-kernel/--half-block)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    if args.impl == "reference":
        return run_reference(args)

    import torch
    from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, Nonbonded

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("gloo")
    torch.cuda.set_device(local)

    t0 = time.perf_counter()
    reps = build_workload(rank, args.replicas)
    natoms = sum(s.npt for s in reps)
    log(f"workload: {len(reps)} replicas, {natoms} atoms, generated in {time.perf_counter() - t0:.1f} s")
    shape = {"water_kernel": {"auto": 0, "full": 1, "half": 2}[args.water_kernel], "half_block": args.half_block}
    forced = args.groups != 0 or args.water_kernel != "auto" or args.half_block != 0
    cache = os.path.join(ROOT, "moil_fnrfd_gb300", "_build", "tune_cache.tsv")
    t0 = time.perf_counter()
    nb = Nonbonded(reps, precision=MOIL_NB_MIXED, device=local, skin=SKIN, list_period=LIST_PERIOD,
                   groups=args.groups, shape=shape, tune_cache=None if forced else cache)
    log(f"handle built in {time.perf_counter() - t0:.1f} s")
    stream = torch.cuda.ExternalStream(nb.stream())
    coor = np.ascontiguousarray(np.concatenate([s.coor for s in reps]), dtype=np.float64)
    d_coor = torch.from_numpy(coor).to(f"cuda:{local}")
    d_dpot = torch.empty_like(d_coor)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=f"cuda:{local}")
    torch.cuda.synchronize()

    def step_device():
        nb.eforce_device(d_coor.data_ptr(), d_dpot.data_ptr(), want_energies=False)

    # kernel and list shapes chosen on this batch by the library's autotuner (coordinate
    # descent over replica groups, water kernel and row build; 2 list periods per candidate)
    tune = None
    if not forced and not args.no_tune:
        t0 = time.perf_counter()
        tune = nb.autotune(d_coor.data_ptr(), d_dpot.data_ptr(), evals=2 * LIST_PERIOD)
        tune["seconds"] = time.perf_counter() - t0
        log(f"autotune: {tune['best']} in {tune['seconds']:.1f} s")
        stream = torch.cuda.ExternalStream(nb.stream())

    for _ in range(args.warmup):
        step_device()
    # per-stage times (library events on its own stream), outside the timed region
    nb.set_timing(True)
    stages = []
    for _ in range(LIST_PERIOD):
        step_device()
        stages.append(nb.timing())
    nb.set_timing(False)
    site_pairs = nb.pair_stats()["site_pairs"]
    launches = int(statistics.median(t["launches"] for t in stages))

    # timed region: device-resident inputs, L2 flushed between steps (not timed)
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    clocks = ClockSampler(local)
    clocks.start()
    ev = []
    for _ in range(args.steps):
        with torch.cuda.stream(stream):
            flush.zero_()
            a = torch.cuda.Event(enable_timing=True)
            b = torch.cuda.Event(enable_timing=True)
            a.record(stream)
        step_device()
        b.record(stream)
        ev.append((a, b))
    torch.cuda.synchronize()
    clk = clocks.stop()
    step_ms = [a.elapsed_time(b) for a, b in ev]
    value, total_s = job_rate(natoms * args.steps, sum(step_ms) / 1e3)

    # e2e through the public host-buffer call: H2D + evaluation + D2H every step, on a handle
    # tuned for that call (the tuner's host objective: more replica groups hide more of the
    # copies) unless the shape is forced
    nbe, tune_host = nb, None
    if not forced and not args.no_tune:
        t0 = time.perf_counter()
        nbe = Nonbonded(reps, precision=MOIL_NB_MIXED, device=local, skin=SKIN, list_period=LIST_PERIOD,
                        shape=shape, tune_cache=cache, tune_host=True)
        tune_host = nbe.autotune(d_coor.data_ptr(), d_dpot.data_ptr(), evals=2 * LIST_PERIOD)
        tune_host["seconds"] = time.perf_counter() - t0
        log(f"autotune (host buffers): {tune_host['best']} in {tune_host['seconds']:.1f} s")
    h_coor = torch.from_numpy(coor).pin_memory()
    h_dpot = torch.empty_like(h_coor).pin_memory()
    hc, hd = h_coor.numpy(), h_dpot.numpy()
    for _ in range(3):
        nbe.eforce_into(hc, hd, want_energies=False)
    torch.cuda.synchronize()
    e2e_ms = []
    for _ in range(args.steps):
        with torch.cuda.stream(stream):
            flush.zero_()
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        nbe.eforce_into(hc, hd, want_energies=False)
        e2e_ms.append((time.perf_counter() - t1) * 1e3)
    e2e_value, _ = job_rate(natoms * args.steps, sum(e2e_ms) / 1e3)
    e2e_shape = nbe.shape()

    press = press_leg(nbe, reps, hc, e2e_ms) if not args.no_press and rank == 0 else None
    if nbe is not nb:
        nbe.close()

    # dominant kernel and its roofline (FP32 pipe): average over steps without a rebuild
    no_build = [t for t in stages if not t["list_rebuilt"]] or stages
    keys = ["water_ms", "atom_ms", "excl_ms", "pme_spread_fft_ms", "pme_conv_ms", "pme_gather_ms", "finalize_ms"]
    avg = {k: statistics.mean(t[k] for t in no_build) for k in keys}
    # prepare_ms: status upload and coordinate conversion, with the skin check folded in (every
    # evaluation); list_ms: the rebuild kernels (amortised over all steps, and per rebuild)
    avg["prepare_ms"] = statistics.mean(t["prepare_ms"] for t in stages)
    avg["list_ms"] = statistics.mean(t["list_ms"] for t in stages)
    built = [t for t in stages if t["list_rebuilt"]]
    if built:
        avg["list_rebuild_ms"] = statistics.mean(t["list_ms"] for t in built)
    if len(built) < len(stages):
        avg["list_check_ms"] = statistics.mean(t["prepare_ms"] for t in stages if not t["list_rebuilt"])
    dom = max(keys, key=lambda k: avg[k])
    sm_mhz = clk["sm_mhz"] or peaks().get("sm_max_mhz", 2070.0)
    peak_fp32 = fp32_peak_tflops(peaks().get("sm_max_mhz", 2070.0))
    # both rooflines (the real-space kernel is the dominant one; PME by its HBM model)
    achieved = site_pairs * F_PAIR / (avg["water_ms"] + avg["atom_ms"]) / 1e9   # TFLOP/s
    n_wat = sum(s.nwaters for s in reps)
    wk = nb.shape()["water_kernel"]
    roof_rs = {"kernel": f"{WATER_KERNEL_NAME[wk]} + k_atom_f (real space)", "bound": "fp32", "achieved": achieved,
               "peak": peak_fp32, "unit": "TFLOP/s", "frac": achieved / peak_fp32,
               "traffic": WATER_KERNEL_DRAM_BYTES_PER_WATER[wk] * n_wat,
               "traffic_note": "bytes per evaluation of the water kernel (all groups): ncu DRAM read+write per "
                               "water on a 48-replica capture x waters",
               "peak_source": "nominal FP32 FMA peak at the measured max SM clock (152 SMs x 128 lanes x 2); "
                              "MEASURED_PEAKS.json has no FP32 figure",
               "work": f"{site_pairs} unique in-cutoff site pairs x {F_PAIR} FP32 ops per launch"}
    hbm = peaks().get("hbm_gbs", 6800.0)
    ng = sum(s.nfft[0] * s.nfft[1] * s.nfft[2] for s in reps)
    b = 56 * natoms + 64 * ng
    t_pme = (avg["pme_spread_fft_ms"] + avg["pme_conv_ms"] + avg["pme_gather_ms"]) / 1e3
    traffic_pme = PME_DRAM_BYTES_PER_ATOM * natoms
    roof_pme = {"kernel": "PME (spread+FFT, convolution, gather)", "bound": "hbm",
                "achieved": b / t_pme / 1e9, "peak": hbm, "unit": "GB/s", "frac": b / t_pme / 1e9 / hbm,
                "traffic": traffic_pme,
                "traffic_note": "ncu DRAM read+write of the five PME kernels per atom on a 48-replica capture "
                                "(cold caches) x atoms; measured DRAM rate at the stage times: "
                                f"{traffic_pme / t_pme / 1e9:.0f} GB/s",
                "peak_source": "MEASURED_PEAKS.json hbm_gbs (measured)",
                "work": f"56 N + 64 Ng bytes per evaluation = {b} B"}
    roof = roof_rs if dom in ("water_ms", "atom_ms") else roof_pme

    out = {"metric": METRIC, "value": value, "unit": "atom-evals/s", "n_gpus": world, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": 1e3 * total_s / args.steps, "higher_is_better": True,
           "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
           "config": {"workload": "512 batched uneven TIP3P boxes (config 3 shape): 1500-12000 atoms each, "
                                  "rc 9 Å, alpha 0.35, PME order 4 on 2/3/5-smooth grids >= 1 pt/Å",
                      "replicas": len(reps), "atoms": natoms, "list_period": LIST_PERIOD, "skin": SKIN,
                      "replica_groups": nb.groups(), "shape": nb.shape(),
                      "l2": "256 MB buffer written between timed steps (untimed)",
                      "precision": "FP32 pair/spline/FFT math, int64 fixed-point forces, FP64 energies and corrections"},
           "stage_ms": {k: round(v, 4) for k, v in avg.items()},
           "site_pairs": site_pairs,
           "roofline": roof,
           "roofline_pme": roof_pme,
           "e2e": {"value": e2e_value, "unit": "atom-evals/s", "h2d_bytes_per_step": int(coor.nbytes),
                   "d2h_bytes_per_step": int(coor.nbytes + 16 * 8 * len(reps)), "shape": e2e_shape},
           "clocks": clk, "gpu_launches": launches * args.steps}
    if tune is not None:
        out["autotune"] = tune
    if tune_host is not None:
        out["autotune_host"] = tune_host

    # energy and gradient errors of the batched evaluation against the oracle (FP64, MOIL's
    # predicate) on a sample of replicas spread over the batch
    if not args.no_cpu and rank == 0:
        out["accuracy_vs_oracle"] = accuracy_leg(nb, reps, d_coor, d_dpot)

    # accuracy and the plain FP64 path on a sample of replicas (denominator of the 20x target)
    if not args.no_fp64 and rank == 0:
        sample = reps[:24]
        d_mixed = d_dpot.cpu().numpy()
        offs = np.cumsum([0] + [s.npt for s in reps])
        errs, fp_ms, fp_atoms = [], 0.0, 0
        for k, s in enumerate(sample):
            p = Nonbonded(s, precision=MOIL_NB_FP64, device=local, skin=SKIN, list_period=LIST_PERIOD)
            st = torch.cuda.ExternalStream(p.stream())
            dc = torch.from_numpy(s.coor).to(f"cuda:{local}")
            dd = torch.empty_like(dc)
            for _ in range(2):
                p.eforce_device(dc.data_ptr(), dd.data_ptr())
            a = torch.cuda.Event(enable_timing=True)
            b = torch.cuda.Event(enable_timing=True)
            a.record(st)
            for _ in range(LIST_PERIOD):
                p.eforce_device(dc.data_ptr(), dd.data_ptr())
            b.record(st)
            torch.cuda.synchronize()
            fp_ms += a.elapsed_time(b)
            fp_atoms += s.npt * LIST_PERIOD
            ref = dd.cpu().numpy()
            mine = d_mixed[offs[k]:offs[k + 1]]
            errs.append(float(np.sqrt(((mine - ref) ** 2).sum() / (ref ** 2).sum())))
            p.close()
        fp64_value = fp_atoms / (fp_ms / 1e3)
        out["plain_fp64"] = {"value": fp64_value, "unit": "atom-evals/s",
                             "sample": f"{len(sample)} replicas of {min(s.npt for s in sample)}-"
                                       f"{max(s.npt for s in sample)} atoms ({sum(s.npt for s in sample)} in all), "
                                       f"one per handle/launch sequence, {LIST_PERIOD} evaluations each "
                                       f"(one list build)",
                             "note": "the FP64 water kernel (a warp per water, each pair once) is bound by the "
                                     "FP64 pipe, 1/64 of the FP32 rate; the 96,000-atom FP64 rate is "
                                     "in single_system_md.plain_fp64_atom_evals_per_s"}
        out["speedup_vs_plain_fp64"] = value / fp64_value
        out["force_err_vs_fp64"] = {"max_rel_rms": max(errs), "replicas": len(errs)}
    nb.close()
    if press is not None:
        out["pressure_analysis"] = press

    if not args.no_adj and rank == 0:
        out["adjoint_64"] = adjoint_leg(local)

    if not args.no_md and rank == 0:
        out["single_system_md"] = md_leg(local)
        out["speedup_vs_plain_fp64_96k"] = value / out["single_system_md"]["plain_fp64_atom_evals_per_s"]

    if not args.no_cpu and rank == 0:
        out["cpu_baseline"] = cpu_baseline(reps)
    if rank == 0:
        print(json.dumps(out), flush=True)


if __name__ == "__main__":
    main()
