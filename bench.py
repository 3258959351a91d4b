"""Benchmark: decorrelated samples/s of GTO-VMC, H2O cc-pVDZ-shaped, 65,536 walkers.

One step = one sweep of all walkers: every electron proposes a single-electron
Gaussian move (exact Metropolis acceptance, Sherman-Morrison inverse update),
then the local energy of every walker is evaluated and reduced.  A full FP64
LU refresh of each inverse runs every 50 sweeps inside the timed region.
Default path: one fused persistent launch per 50 sweeps (refresh, moves,
local energies; the batched entry points with one molecule), the timed
launches replayed from a CUDA graph; --path split runs oqmc_sweeps (moves and
local energies of 50 sweeps in one launch) and the refresh between its calls.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--precision mixed|fp64] [--system H2O] [--walkers 65536]
                    [--path persistent|split]
                    [--workload h2o|batched|learned|alle|h2|lih]

value     = walkers x sweeps/s / tau_int(E_L)  (decorrelated samples/s, all ranks)
tau_int   = kappa of the reference's do_binning_analysis (OmegaQMC/utils.py:86-150)
            on the walker-mean E_L series (sweeps); from the timed series when it
            has >= 1000 sweeps, else from an untimed 2000-sweep run.
e2e       = the same metric through the public API with host buffers: every call
            copies the walker positions host->device (pinned), runs its sweeps
            (50 per call on the persistent path, 1 on the split path) and copies
            positions + the reductions back.
--impl reference  times the reference algorithm (all-electron moves, log|psi|
            recomputed twice per step, E_L every step) restated in C/OpenMP on
            all host cores.
Multi-GPU: one process per GPU, independent walker sets (replicas; no
collective on the data path), value summed over ranks, time = max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

REFRESH_EVERY = 50


def binning_analysis(series):
    """(mean, serr, sdev, kappa) of the reference's do_binning_analysis
    (OmegaQMC/utils.py:86-150), the package's copy the VMC driver uses."""
    from omegaqmc_b200.vmc import binning_analysis as ba
    return ba(series)

EQUIL_SWEEPS = 3000
SCALED_R0, SCALED_FMIN = 1.0, 0.05
# nucleus-scaled proposal of the persistent headline path (chosen by measured
# tau_int on H2O: fmin 0.02 and acceptance 0.5 gave tau 1.5 sweeps, against
# 2.4 for fmin 0.05 and 4.1 at the reference's 0.4 target)
HEAD_R0, HEAD_FMIN, HEAD_ACC = 1.0, 0.02, 0.5
# the headline's timed region lasts at least this long (s); its sweep count
# is capped by the measurement buffer
MIN_TIMED_S = 2.0
# chunks of the end-to-end leg's overlapped walker copies
E2E_CHUNKS = 4
MAX_TIMED_SWEEPS = 60000
# the plain FP64 sampler's tau_int (several hundred sweeps) comes from this
# many consecutive segments of PLAIN_SEG sweeps: their kappas give the spread
PLAIN_SEGS, PLAIN_SEG = 4, 12500
# and is cross-checked on PLAIN_TRACE_W walkers' own E_L series of
# PLAIN_TRACE_SWEEPS sweeps
PLAIN_TRACE_W, PLAIN_TRACE_SWEEPS = 1024, 20000


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10000)
    ap.add_argument("--warmup", type=int, default=200)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--precision", default="mixed", choices=["mixed", "fp64"])
    ap.add_argument("--system", default="H2O")
    ap.add_argument("--walkers", type=int, default=65536)
    ap.add_argument("--step-size", type=float, default=0.0)
    ap.add_argument("--cpu-seconds", type=float, default=15.0)
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--proposal", default="scaled", choices=["scaled", "plain"])
    ap.add_argument("--eloc", default="cc", choices=["cc", "tc"],
                    help="local energy on CUDA cores (specialised) or tensor cores (tcgen05)")
    ap.add_argument("--workload", default="h2o",
                    choices=["h2o", "batched", "learned", "alle", "h2", "lih"],
                    help="h2o: the headline H2O metric; batched: H2, LiH, H2O, N2 and "
                         "(H2O)2 in one persistent launch under a CUDA graph; learned: N2 "
                         "with the trained MLP proposal against the plain random walk; "
                         "alle: the reference's all-electron move; h2, lih: "
                         "the H2/STO-3G plain-method workload (FP64, 1,024 walkers) and the "
                         "LiH workload (16,384 walkers, FP64 against mixed, with "
                         "per-output errors)")
    ap.add_argument("--path", default="persistent", choices=["persistent", "split"],
                    help="persistent: one fused launch per 50 sweeps (refresh, moves, E_L) "
                         "under a CUDA graph; split: oqmc_sweeps (moves and E_L of 50 sweeps "
                         "in one launch, refresh in its own)")
    ap.add_argument("--quick", action="store_true",
                    help="profiling mode: no equilibration, comparison, e2e or CPU legs")
    ap.add_argument("--generic", action="store_true",
                    help="split path only: the table-driven kernels (no per-molecule NVRTC "
                         "specialisation), the library's path where NVRTC is absent")
    return ap.parse_args()


STEP_DEFAULT = {"H2": 0.6, "LiH": 0.5, "H2O": 0.3, "N2": 0.3, "H2O_dimer": 0.3}


def build_system(name):
    from omegaqmc_b200 import molecules as M
    from omegaqmc_b200.system import build_system as bs
    mf = M.make_mf(name)
    return bs(mf, M.benchmark_params_corr(mf.mol))


def work_per_walker_sweep(s, acc=0.5):
    """Algorithmic work of one sweep of one walker (FMA = 2 flops).

    Moves (per electron): distinct exponentials; radial sums 2 flops per
    (primitive, column); angular 3 (p) / 17 (d) / 12*(2l+1) (f, g); MO row
    2 per MO coefficient; ratio vector 2 nocc^2; Sherman-Morrison 2 nocc^2 x
    acceptance; Jastrow change 2 x 14 flops per other particle.  Local
    energy (per electron): exponentials; radial VGL 6 flops per (primitive,
    column); angular VGL 12 per AO; MO VGL 10 per MO coefficient; Slater
    assembly 8 nocc + 6; Jastrow VGL 20 per partner; Coulomb 10 per pair.
    The MO coefficients counted are those the generated kernels evaluate
    (``mo_terms``); ``flops_dense`` counts all nbf x nocc of them.
    """
    groups = s.prim_groups()
    n_exp = sum(len(a) for _, a, _ in groups)
    rad = sum(len(a) * len(ids) for _, a, ids in groups)
    ang_v = sum({0: 0, 1: 3, 2: 17}.get(sh.am, 12 * (2 * sh.am + 1)) for sh in s.shells)
    ne, no, nb, nn = s.n_e, s.nocc, s.nbf, s.natm

    def total(nc):
        move = 2 * rad + ang_v + 2 * nc + 2 * no * no + 2 * no * no * acc + 28 * (ne - 1 + nn)
        el = 6 * rad + 12 * nb + 10 * nc + 8 * no + 6 + 20 * (ne - 1 + nn)
        coul = 10 * (ne * (ne - 1) // 2 + ne * nn)
        return float(ne * (move + el) + coul)

    return {"flops": total(mo_terms(s)), "flops_dense": total(nb * no),
            "mo_terms": mo_terms(s), "exps": float(2 * ne * n_exp)}


def mo_terms(s):
    """MO coefficients the generated kernels evaluate: those above 1e-12 of
    their orbital's largest |coefficient| (the kernel generator leaves out
    the round-off-level entries that point-group symmetry makes zero)."""
    C = np.abs(np.asarray(s.C, dtype=np.float64))
    cmax = C.max(axis=0, keepdims=True)
    return int(np.count_nonzero((C != 0.0) & (C > 1e-12 * cmax)))


class ClockSampler:
    """nvidia-smi clocks/throttle sampling during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.rows = []
        self.first = 0
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
            # nvidia-smi takes a moment to start: wait for its first row so
            # that the rows kept (those after it) fall inside the timed region
            t0 = time.perf_counter()
            while not self.rows and time.perf_counter() - t0 < 3.0 and self.proc.poll() is None:
                time.sleep(0.01)
            self.first = len(self.rows)
        except FileNotFoundError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        rows = self.rows[self.first:] or self.rows
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4)
                          if len(r) > 5 + k and r[5 + k].lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons,
                "samples": len(rows)}


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def cpu_reference(system, seconds, nthreads, step, seed=7, n_equil=300):
    """Reference algorithm on host cores (OmegaQMC/vmc_gto.py:1338-1357 step
    adaptation during equilibration, then fixed-step production); returns
    (walker-steps/s, tau_int, acceptance, sample description, E_L series)."""
    from oracle import cref
    from omegaqmc_b200.sampler import init_walkers_gaussian
    W = 256
    X = np.ascontiguousarray(init_walkers_gaussian(system, W, 1.0, seed))
    for k in range(n_equil):
        _, acc = cref.run(system, X, 1, step, seed=seed * 1000003 + k, nthreads=nthreads)
        step = float(np.exp(np.log(step) + 0.05 * (acc - 0.4)))
    t0 = time.perf_counter()
    cref.run(system, X, 10, step, seed=seed + 1, nthreads=nthreads)
    per_step = (time.perf_counter() - t0) / 10
    n = max(200, int(seconds / max(per_step, 1e-6)))
    t0 = time.perf_counter()
    ser, acc = cref.run(system, X, n, step, seed=seed + 2, nthreads=nthreads)
    dt = time.perf_counter() - t0
    rate = W * n / dt
    _, _, _, kappa = binning_analysis(ser[:, 3])
    return (rate, kappa, acc,
            f"{W} walkers x {n} steps ({dt:.1f} s) after {n_equil} adaptive equilibration "
            f"steps, step {step:.3f}", ser[:, 3])


def output_errors(ctx, X, precision, step, seed):
    """Error of every per-walker output the sampler works with
    (oqmc_state_eval: tracked log|psi|, grad log|psi|, per-electron
    Laplacian, E_L) against the FP64 evaluation at the same positions
    (oqmc_eval, itself matched to the oracle at 1e-10), on the given
    configurations: right after the FP64 LU refresh, and after 49 sweeps of
    Sherman-Morrison updates (the longest stretch between refreshes).
    Errors: |d| for log|psi| and E_L (Ha); |d| / (|x| + 1) for each
    gradient component and Laplacian.  Returns max / p99 / median each."""
    from omegaqmc_b200.sampler import WalkerEnsemble
    out = {"walkers": int(X.shape[0])}
    for sweeps in (0, 49):
        ens = WalkerEnsemble(ctx, X, precision, seed=seed, refresh_every=10**9)
        if sweeps:
            ens.run(sweeps, step)
        got = ens.state_evaluate()
        ref = ctx.evaluate(ens.X)
        errs = {"logpsi": (got["logpsi"] - ref["logpsi"]).abs(),
                "grad": (got["grad"] - ref["grad"]).abs() / (ref["grad"].abs() + 1),
                "lap": (got["lap"] - ref["lap"]).abs() / (ref["lap"].abs() + 1),
                "e_loc": (got["e_loc"] - ref["e_loc"]).abs()}
        st = {}
        for k, v in errs.items():
            v = v.reshape(-1).cpu().numpy()
            st[k] = {"max": float(v.max()), "p99": float(np.quantile(v, 0.99)),
                     "median": float(np.median(v))}
        out[f"after_{sweeps}_sweeps"] = st
        del ens
    return out


def walker_series_kappa(ctx, X, step, seed, sweeps=None):
    """Cross-check of a long tau_int: kappa of the reference's estimator on
    each walker's own E_L series (W walkers, the given sweeps, FP64, the
    context's proposal), averaged over the walkers with its standard error.
    Walkers are independent, so each series has the tau_int of the
    walker-mean series; the average of many short-series estimates is far
    less noisy than one estimate on the mean series."""
    import torch
    from omegaqmc_b200.sampler import NSUM, WalkerEnsemble
    sweeps = sweeps or PLAIN_TRACE_SWEEPS
    W = int(X.shape[0])
    ens = WalkerEnsemble(ctx, X, "fp64", seed=seed)
    trace = torch.empty(sweeps, W, dtype=torch.float64, device=X.device)
    sums = torch.zeros(sweeps, NSUM, dtype=torch.float64, device=X.device)
    ens.run(sweeps, step, sums=sums, el_trace=trace)
    tr = trace.cpu().numpy()
    ks = np.array([binning_analysis(tr[:, w])[3] for w in range(W)])
    del ens, trace
    return {"walkers": W, "sweeps": sweeps, "mean": float(ks.mean()),
            "serr": float(ks.std(ddof=1) / np.sqrt(W)), "median": float(np.median(ks))}


def kappa_spread(series, parts):
    """kappa of each of `parts` consecutive segments of a series: their mean
    and standard error (the uncertainty of a tau_int estimate)."""
    n = len(series) // parts
    ks = [binning_analysis(series[i * n:(i + 1) * n])[3] for i in range(parts)]
    return {"segments": parts, "segment_sweeps": n, "kappas": ks,
            "mean": float(np.mean(ks)), "serr": float(np.std(ks, ddof=1) / np.sqrt(parts))}


def sweep_launches(ens, n_sweeps, measure_every=1):
    """Kernels that ``ens.run(n_sweeps)`` launches with the learned proposal from
    the ensemble's current refresh phase (the chunking of WalkerEnsemble.run): per oqmc_sweeps call a
    layout conversion in and one out, per measurement a move kernel and a
    local-energy kernel (one more move kernel for sweeps after the last
    measurement of a call), per FP64 refresh a conversion and the refresh
    kernel."""
    since, n, done = ens.since_refresh, 0, 0
    while done < n_sweeps:
        chunk = min(n_sweeps - done, ens.refresh_every - since)
        if measure_every > 1:
            chunk = max(measure_every, chunk - chunk % measure_every)
            chunk = min(chunk, n_sweeps - done)
        m = chunk // measure_every
        n += 2 + 2 * m + (1 if chunk > m * measure_every else 0)
        done += chunk
        since += chunk
        if since >= ens.refresh_every:
            n += 2
            since = 0
    return n


def fused_launches(ens, n_sweeps, measure_every=1, tensor_core_energy=False):
    """Kernels that ``ens.run(n_sweeps)`` launches where the sweeps are fused
    (single-electron sweeps and FP64 all-electron steps): one per oqmc_sweeps
    call, or with the tensor-core local energy a sweep and an energy kernel
    per measurement (one more sweep kernel for sweeps after the last
    measurement of a call); per FP64 refresh a conversion and the refresh
    kernel."""
    since, n, done = ens.since_refresh, 0, 0
    while done < n_sweeps:
        chunk = min(n_sweeps - done, ens.refresh_every - since)
        if measure_every > 1:
            chunk = max(measure_every, chunk - chunk % measure_every)
            chunk = min(chunk, n_sweeps - done)
        m = chunk // measure_every
        n += 2 * m + (1 if chunk > m * measure_every else 0) if tensor_core_energy else 1
        done += chunk
        since += chunk
        if since >= ens.refresh_every:
            n += 2
            since = 0
    return n


def split_launches(ens, n_sweeps, generic, tensor_core_energy):
    """Kernels that ``ens.run(n_sweeps)`` launches on the split path (E_L every
    sweep).  Above 37,888 walkers a walker has one thread: table-driven sweeps
    of four and more orbitals then move in a kernel of their own, as the learned
    proposal's do, and FP64 ensembles of eight and more have their local
    energies in one."""
    one = ens.W > 148 * 256
    if generic and one and ens.ctx.nocc >= 4:
        return sweep_launches(ens, n_sweeps)
    apart = one and not generic and ens.precision == "fp64" and ens.ctx.nocc >= 8
    return fused_launches(ens, n_sweeps, 1, tensor_core_energy or apart)


def adapt_step(ens, step, n_chunks=40, chunk=5, target=0.4):
    """Equilibrate with the reference's rule log s += 0.05 (acc - target)
    applied once per chunk of sweeps (OmegaQMC/vmc_gto.py:121-126)."""
    for _ in range(n_chunks):
        s = ens.run(chunk, step).cpu().numpy()
        acc = s[:, 5].sum() / (chunk * ens.W * ens.ctx.n_e)
        step = float(np.exp(np.log(step) + 0.05 * 5 * (acc - target)))
    return step


def run_reference(a):
    rank, world, _ = dist_env()
    if rank != 0:
        return
    system = build_system(a.system)
    step = a.step_size or STEP_DEFAULT.get(a.system, 0.3) * 1.0
    cores = len(os.sched_getaffinity(0))
    # initial step of the reference's adaptation (sqrt(3 * mc_timestep))
    ref_step = (3 * 0.1) ** 0.5
    rates, kappas = [], []
    for _ in range(max(1, min(a.steps, 3))):
        rate, kappa, acc, sample, _ = cpu_reference(system, a.cpu_seconds / 3, cores, ref_step)
        rates.append(rate)
        kappas.append(kappa)
    rate = float(np.mean(rates))
    kappa = float(np.mean(kappas))
    value = rate / kappa
    unit = "decorrelated samples/s"
    line = {
        "impl": "reference",
        "metric": "decorrelated samples/s (walker-steps/s / tau_int) vs plain FP64, H2O 64k walkers",
        "value": value, "unit": unit, "n_gpus": world, "steps": a.steps, "warmup": a.warmup,
        "ms_per_step": 256 / rate * 1e3, "higher_is_better": True, "scaling": "weak",
        "dtype": "f64", "data": "synthetic",
        "config": {"workload": f"{a.system} cc-pVDZ-shaped, 256 walkers per timed sample on "
                               f"{cores} host threads, all-electron Gaussian steps (the "
                               "reference's move) + E_L every step, FP64, no refresh (every "
                               "step recomputes log|psi| afresh)",
                   "reference_path": "the reference algorithm (all-electron Gaussian moves, "
                                     "log|psi| recomputed twice per step, E_L every step) in "
                                     f"C/OpenMP on {cores} host threads",
                   "reference_sample": "256 walkers per timed sample (the walker-step rate "
                                       "does not depend on the walker count)",
                   "step": ref_step},
        "walker_steps_per_s": rate, "tau_int": kappa, "acceptance": acc,
        "cpu_baseline": {"value": value, "unit": unit, "cores": cores, "kind": "port",
                         "sample": sample},
        "e2e": {"value": value, "unit": unit, "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
        "vs_baseline": None,
    }
    print(json.dumps(line), flush=True)


def run_ours(a):
    import torch
    import torch.distributed as dist
    from omegaqmc_b200 import _lib as L
    from omegaqmc_b200.context import GTOContext
    from omegaqmc_b200.sampler import WalkerEnsemble, init_walkers_gaussian, NSUM

    rank, world, local = dist_env()
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    system = build_system(a.system)
    ctx = GTOContext(system)
    t_spec = time.perf_counter()
    if not a.generic:
        ctx.specialize()             # NVRTC-compiled kernels for this molecule
    t_spec = time.perf_counter() - t_spec
    if a.proposal == "scaled":
        ctx.set_proposal(1, SCALED_R0, SCALED_FMIN)
    if a.eloc == "tc" and a.precision == "mixed":
        ctx.use_tensor_cores(True)
    W = a.walkers
    step = a.step_size or STEP_DEFAULT.get(a.system, 0.3)
    X0 = init_walkers_gaussian(system, W, 1.0, seed=1000 + rank)
    ens = WalkerEnsemble(ctx, X0, a.precision, seed=2024 + 7919 * rank,
                         refresh_every=REFRESH_EVERY)
    stream = torch.cuda.current_stream()

    # set-up: step adaptation and a fixed equilibration (core electrons start
    # far from their equilibrium density), then the W warm-up sweeps
    if a.quick:
        a.no_e2e = a.no_cpu = True
        step = a.step_size or 0.8
    else:
        if not a.step_size:
            step = adapt_step(ens, step)
        ens.run(EQUIL_SWEEPS, step)
    ens.run(max(a.warmup, 3), step)
    torch.cuda.synchronize()

    K = a.steps
    sums = torch.zeros(K, NSUM, dtype=torch.float64, device=dev)
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    n_launch = split_launches(ens, K, a.generic, a.eloc == "tc" and a.precision == "mixed")
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        ev0.record(stream)
        ens.run(K, step, sums=sums)
        ev1.record(stream)
        torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    ms = ev0.elapsed_time(ev1)
    flags = ctx.flags()
    s_np = sums.cpu().numpy()
    series = s_np[:, 3] / np.maximum(s_np[:, 6], 1)
    if K >= 1000 or a.quick:
        tau_series = series
        tau_src = f"timed series ({K} sweeps)"
    else:
        aux = ens.run(2000, step).cpu().numpy()
        tau_series = aux[:, 3] / np.maximum(aux[:, 6], 1)
        tau_src = "untimed 2000-sweep series"
    e_mean, e_serr, e_sdev, kappa = binning_analysis(tau_series)
    acc = float(s_np[:, 5].sum() / (K * W * system.n_e))

    # the comparison target: the plain FP64 sampler on the same walkers
    plain = None
    if not a.quick and (a.precision != "fp64" or a.proposal != "plain"):
        pctx = GTOContext(system)            # fixed-width Gaussian proposal
        pctx.specialize()
        pe = WalkerEnsemble(pctx, ens.X, "fp64", seed=99 + rank, refresh_every=REFRESH_EVERY)
        pstep = adapt_step(pe, STEP_DEFAULT.get(a.system, 0.3))
        pe.run(500, pstep)
        Kp = 4000
        ps = torch.zeros(Kp, NSUM, dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        p0 = torch.cuda.Event(enable_timing=True)
        p1 = torch.cuda.Event(enable_timing=True)
        p0.record(stream)
        pe.run(Kp, pstep, sums=ps)
        p1.record(stream)
        torch.cuda.synchronize()
        pms = p0.elapsed_time(p1)
        pn = ps.cpu().numpy()
        pser = pn[:, 3] / np.maximum(pn[:, 6], 1)
        pm, pse, _, pk = binning_analysis(pser)
        pw = W * Kp / (pms * 1e-3)
        plain = {"value": pw * world / pk, "walker_sweeps_per_s": pw * world, "tau_int": pk,
                 "proposal": "fixed-width Gaussian", "step": pstep,
                 "ms_per_step": pms / Kp, "steps": Kp,
                 "energy": {"mean": pm, "serr": pse},
                 "energy_diff_sigma": abs(pm - e_mean) / max(np.hypot(pse, e_serr), 1e-300)}
        del pe

    # kernel-level timing of the dominant kernel on its own stream: one chunk
    # of REFRESH_EVERY sweeps = one oqmc_sweeps call; the refresh separately
    chunk_sums = torch.zeros(REFRESH_EVERY, NSUM, dtype=torch.float64, device=dev)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e2 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    ctx.sweeps(ens.X, ens.state, ens.prec, REFRESH_EVERY, step, ens.seed, 10**7,
               chunk_sums, stream=stream)
    e1.record(stream)
    ctx.refresh(ens.X, ens.state, ens.prec, stream=stream)
    e2.record(stream)
    torch.cuda.synchronize()
    sweep_ms = e0.elapsed_time(e1)
    refresh_ms = e1.elapsed_time(e2)

    # e2e: host buffers through the public API
    e2e = None
    if not a.no_e2e:
        Ke = min(K, 200)
        hostX = torch.empty_like(ens.X, device="cpu").pin_memory()
        hostX.copy_(ens.X)
        host_sums = torch.empty(NSUM, dtype=torch.float64).pin_memory()
        s1 = torch.zeros(Ke, NSUM, dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        f0 = torch.cuda.Event(enable_timing=True)
        f1 = torch.cuda.Event(enable_timing=True)
        f0.record(stream)
        for k in range(Ke):
            ens.X.copy_(hostX, non_blocking=True)
            ens.run(1, step, sums=s1[k:k + 1])
            hostX.copy_(ens.X, non_blocking=True)
            host_sums.copy_(s1[k], non_blocking=True)
        f1.record(stream)
        torch.cuda.synchronize()
        ems = f0.elapsed_time(f1)
        bi = ens.X.numel() * 8
        e2e = {"ms_per_step": ems / Ke, "steps": Ke,
               "h2d_bytes_per_step": bi, "d2h_bytes_per_step": bi + NSUM * 8}

    # max over ranks
    t = torch.tensor([ms, e2e["ms_per_step"] if e2e else 0.0], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_max, e2e_ms = float(t[0]), float(t[1])

    wss = W * world * K / (ms_max * 1e-3)
    value = wss / kappa
    work = work_per_walker_sweep(system, acc)
    if a.generic:   # the table-driven kernels evaluate every MO coefficient
        work["flops"], work["mo_terms"] = work["flops_dense"], system.nbf * system.nocc
    peak_kind = 0 if a.precision == "fp64" else 1
    rate = ctypes_peak(L, peak_kind)
    achieved = work["flops"] * W * REFRESH_EVERY / (sweep_ms * 1e-3)
    traffic = None if a.generic else ncu_traffic(a.system, a.precision)
    line = {
        "metric": "decorrelated samples/s (walker-steps/s / tau_int) vs plain FP64, H2O 64k walkers",
        "value": value, "unit": "decorrelated samples/s", "n_gpus": world, "steps": K,
        "steps_requested": a.steps,
        "steps_note": f"the timed region replays whole 50-sweep launches for at least "
                      f"{MIN_TIMED_S:g} s: {K} sweeps",
        "warmup": a.warmup, "ms_per_step": ms_max / K, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "f32+f64" if a.precision == "mixed" else "f64",
        "data": "synthetic",
        "config": {"workload": f"{a.system} cc-pVDZ-shaped, {W} walkers/GPU, single-electron "
                               f"sweeps + E_L every sweep, FP64 LU refresh every {REFRESH_EVERY}",
                   "precision": a.precision, "walkers_per_gpu": W, "step": step,
                   "parallelism": f"replicas x{world}",
                   "trial": "RHF determinant + Pade J2 (b=3)",
                   "kernels": ("table-driven (generic) kernels" if a.generic else
                               f"NVRTC-specialised to the molecule (compile {t_spec:.1f} s, untimed)"),
                   "local_energy": "tcgen05 tensor cores (split TF32/BF16)" if a.eloc == "tc"
                                   else "CUDA cores",
                   "proposal": (f"nucleus-scaled Gaussian (r0={SCALED_R0}, fmin={SCALED_FMIN}), "
                                "exact MH" if a.proposal == "scaled" else "fixed-width Gaussian"),
                   "equilibration_sweeps": EQUIL_SWEEPS + 200,
                   "l2": "walker state stays in shared memory for a whole launch; "
                         "inputs 41 MB are re-read once per 50-sweep launch"},
        "walker_sweeps_per_s": wss, "tau_int": kappa, "tau_source": tau_src,
        "energy": {"mean": e_mean, "serr": e_serr}, "acceptance": acc, "kernel_flags": flags,
        "gpu_launches": n_launch,
        "roofline": {"bound": "fp64" if peak_kind == 0 else "fp32",
                     "achieved": achieved / 1e12, "peak": rate / 1e12, "unit": "TFLOP/s",
                     "frac": achieved / rate if rate else None, "traffic": traffic,
                     "kernel": ("k_moves and k_eloc" if a.generic else "k_sweeps") +
                               " (one 50-sweep oqmc_sweeps call)",
                     "kernel_ms_per_launch": sweep_ms,
                     "refresh_ms_per_launch": refresh_ms,
                     "flops_per_walker_sweep": work["flops"],
                     "flops_per_walker_sweep_dense": work["flops_dense"],
                     "mo_terms": work["mo_terms"],
                     "peak_source": "own FMA microkernel (oqmc_measure_peak), of measured"},
    }
    if plain:
        line["plain_fp64"] = plain
        line["speedup_vs_plain_fp64"] = value / plain["value"]
    if e2e:
        line["e2e"] = {"value": W * world / (e2e_ms * 1e-3) / kappa,
                       "unit": "decorrelated samples/s",
                       "h2d_bytes_per_step": e2e["h2d_bytes_per_step"],
                       "d2h_bytes_per_step": e2e["d2h_bytes_per_step"],
                       "ms_per_step": e2e_ms}
    if rank == 0 and not a.no_cpu and world == 1:
        cores = len(os.sched_getaffinity(0))
        r, kap, acc_c, sample, _ = cpu_reference(system, a.cpu_seconds, cores, (3 * 0.1) ** 0.5)
        line["cpu_baseline"] = {"value": r / kap, "unit": "decorrelated samples/s",
                                "cores": cores, "kind": "port", "sample": sample,
                                "walker_steps_per_s": r, "tau_int": kap}
    line["clocks"] = clk.summary()
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


def run_persistent(a):
    """The headline: one molecule through the fused persistent kernel (the
    batched entry points with a single system).  Each launch = FP64 LU
    refresh + 50 single-electron sweeps with E_L every sweep; the timed
    region replays a CUDA graph of K/50 launches.  The plain FP64 sampler
    (fixed-width Gaussian, the reference's 0.4 acceptance rule) runs through
    the same path for the comparison."""
    import torch
    import torch.distributed as dist
    from omegaqmc_b200 import _lib as L
    from omegaqmc_b200 import replicas as RP
    from omegaqmc_b200.batch import BatchedSampler
    from omegaqmc_b200.context import GTOContext
    from omegaqmc_b200.sampler import WalkerEnsemble, init_walkers_gaussian, NSUM

    rank, world, local = dist_env()
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    system = build_system(a.system)
    ctx = GTOContext(system)
    t_spec = time.perf_counter()
    ctx.specialize()
    W = a.walkers
    K_req = max(REFRESH_EVERY, (a.steps // REFRESH_EVERY) * REFRESH_EVERY)
    cap = max(K_req, MAX_TIMED_SWEEPS, 2000)
    seed = 2024 + 7919 * rank
    scaled = a.proposal == "scaled"
    X0 = init_walkers_gaussian(system, W, 1.0, seed=1000 + rank)
    b = BatchedSampler([ctx], [X0], [a.step_size or 0.8], precision=a.precision,
                       proposal=a.proposal, scale_r0=HEAD_R0, scale_fmin=HEAD_FMIN,
                       cap=cap)
    t_spec = time.perf_counter() - t_spec
    stream = torch.cuda.current_stream()
    EQ1, EQ2, WARM, KERN, E2E = 10**7, 2 * 10**7, 3 * 10**7, 4 * 10**7, 5 * 10**7

    def sweeps_no_meas(n, base):
        b.reset(base)
        for _ in range(max(1, n // REFRESH_EVERY)):
            b.run(REFRESH_EVERY, REFRESH_EVERY + 1, seed)

    if not a.quick:
        sweeps_no_meas(EQUIL_SWEEPS // 3, EQ1)
        if not a.step_size:
            b.adapt_steps(HEAD_ACC if scaled else 0.4, seed=seed ^ 1)
        sweeps_no_meas(2 * EQUIL_SWEEPS // 3, EQ2)
    cfg, _ = b.tune(4, seed=seed ^ 0x55)
    step = b.steps()[0]
    sweeps_no_meas(max(a.warmup, 3), WARM)
    # the timed region replays at least MIN_TIMED_S of launches, whatever
    # --steps asks for: two launches timed alone set the count (the same on
    # every rank: the max over ranks)
    b.reset(KERN)
    q0 = torch.cuda.Event(enable_timing=True)
    q1 = torch.cuda.Event(enable_timing=True)
    q0.record(stream)
    for _ in range(2):
        b.run(REFRESH_EVERY, 1, seed)
    q1.record(stream)
    torch.cuda.synchronize()
    tq = torch.tensor([q0.elapsed_time(q1) / 2], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(tq, op=dist.ReduceOp.MAX)
    n_launch = max(K_req // REFRESH_EVERY,
                   int(np.ceil(MIN_TIMED_S * 1e3 / max(float(tq[0]), 1e-3))))
    n_launch = min(n_launch, cap // REFRESH_EVERY)
    if a.quick:                      # profiling: exactly the launches asked for
        n_launch = K_req // REFRESH_EVERY
    K = n_launch * REFRESH_EVERY
    b.capture(n_launch, REFRESH_EVERY, 1, seed)
    b.reset(0)
    torch.cuda.synchronize()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    if world > 1:
        dist.barrier()
    with ClockSampler(local) as clk:
        torch.cuda.nvtx.range_push("headline_timed")
        ev0.record(stream)
        b.replay()
        ev1.record(stream)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_pop()
    if world > 1:
        dist.barrier()
    ms = ev0.elapsed_time(ev1)
    flags = b.flags()
    # replicas: the measurement sums of all ranks add up to those of the
    # union of their walkers
    s_np = RP.combine_sums(b.sums[0][:K].clone()).cpu().numpy()
    series = RP.walker_mean_series(s_np)
    acc = float(s_np[:, 5].sum() / (K * W * world * system.n_e))
    if K >= 1000 or a.quick:
        tau_series, tau_src = series, f"timed series ({K} sweeps)"
    else:
        b.reset(E2E + 10**6)
        for _ in range(40):
            b.run(REFRESH_EVERY, 1, seed)
        aux = RP.combine_sums(b.sums[0][:2000].clone()).cpu().numpy()
        tau_series = RP.walker_mean_series(aux)
        tau_src = "untimed 2000-sweep series"
    e_mean, e_serr, e_sdev, kappa = binning_analysis(tau_series)
    kq = kappa_spread(tau_series, 4)

    # one launch (refresh + 50 sweeps) timed on its own: the roofline denominator
    b.reset(KERN)
    k0 = torch.cuda.Event(enable_timing=True)
    k1 = torch.cuda.Event(enable_timing=True)
    k0.record(stream)
    b.run(REFRESH_EVERY, 1, seed)
    k1.record(stream)
    torch.cuda.synchronize()
    launch_ms = k0.elapsed_time(k1)

    plain = prec = fp64s = None
    if not a.quick and (a.precision != "fp64" or a.proposal != "plain"):
        # the comparison: plain FP64 sampler through the same path; its
        # tau_int (several hundred sweeps) from PLAIN_SEGS consecutive
        # segments of one chain, PLAIN_SEG sweeps each, all timed
        pb = BatchedSampler([ctx], [b.walkers[0].clone()], [STEP_DEFAULT.get(a.system, 0.3)],
                            precision="fp64", proposal="plain", cap=PLAIN_SEG)
        pstep = pb.adapt_steps(0.4, seed=seed ^ 2)[0]
        pb.reset(EQ1 + 10**6)
        for _ in range(20):
            pb.run(REFRESH_EVERY, REFRESH_EVERY + 1, seed ^ 3)
        pb.tune(4, seed=seed ^ 4)
        pms, pser = 0.0, []
        for seg in range(PLAIN_SEGS):
            pb.reset(seg * PLAIN_SEG)
            p0 = torch.cuda.Event(enable_timing=True)
            p1 = torch.cuda.Event(enable_timing=True)
            p0.record(stream)
            for _ in range(PLAIN_SEG // REFRESH_EVERY):
                pb.run(REFRESH_EVERY, 1, seed ^ 3)
            p1.record(stream)
            torch.cuda.synchronize()
            pms += p0.elapsed_time(p1)
            pn = pb.sums[0][:PLAIN_SEG].cpu().numpy()
            pser.append(pn[:, 3] / np.maximum(pn[:, 6], 1))
        pser = np.concatenate(pser)
        Kp = PLAIN_SEGS * PLAIN_SEG
        pm, pse, _, pk = binning_analysis(pser)
        pks = kappa_spread(pser, PLAIN_SEGS)
        pw = W * Kp / (pms * 1e-3)
        plain = {"value": pw * world / pk, "walker_sweeps_per_s": pw * world, "tau_int": pk,
                 "tau_int_segments": pks,
                 "proposal": "fixed-width Gaussian", "step": pstep, "precision": "fp64",
                 "ms_per_step": pms / Kp, "steps": Kp, "path": "same persistent kernel, FP64",
                 "energy": {"mean": pm, "serr": pse},
                 "energy_diff_sigma": abs(pm - e_mean) / max(np.hypot(pse, e_serr), 1e-300),
                 "tau_int_walker_series": walker_series_kappa(
                     ctx, pb.walkers[0][:PLAIN_TRACE_W], pstep, seed ^ 12)}
        del pb
        # FP64 with the headline's proposal: separates the precision factor
        # (mixed vs FP64, same proposal) from the proposal factor (scaled vs
        # fixed-width, both FP64)
        if a.precision != "fp64" and scaled:
            fb = BatchedSampler([ctx], [b.walkers[0].clone()], [step], precision="fp64",
                                proposal="scaled", scale_r0=HEAD_R0, scale_fmin=HEAD_FMIN,
                                cap=10000)
            fb.adapt_steps(HEAD_ACC, seed=seed ^ 8)
            fb.reset(EQ1 + 3 * 10**6)
            for _ in range(10):
                fb.run(REFRESH_EVERY, REFRESH_EVERY + 1, seed ^ 9)
            fb.tune(4, seed=seed ^ 10)
            Kf = 10000
            fb.reset(0)
            f0 = torch.cuda.Event(enable_timing=True)
            f1 = torch.cuda.Event(enable_timing=True)
            f0.record(stream)
            for _ in range(Kf // REFRESH_EVERY):
                fb.run(REFRESH_EVERY, 1, seed ^ 9)
            f1.record(stream)
            torch.cuda.synchronize()
            fms = f0.elapsed_time(f1)
            fn = fb.sums[0][:Kf].cpu().numpy()
            fser = fn[:, 3] / np.maximum(fn[:, 6], 1)
            fmu, fse, _, fk = binning_analysis(fser)
            fw = W * Kf / (fms * 1e-3)
            fp64s = {"value": fw * world / fk, "walker_sweeps_per_s": fw * world,
                     "tau_int": fk, "tau_int_segments": kappa_spread(fser, 4),
                     "ms_per_step": fms / Kf, "steps": Kf, "step": fb.steps()[0],
                     "proposal": "nucleus-scaled Gaussian (the headline's)", "precision": "fp64",
                     "energy": {"mean": fmu, "serr": fse}}
            del fb
        # precision, paired: the mixed and the FP64 sampler start from the same
        # walkers with the same proposal, step, seed and RNG counters, so they
        # take the same decisions until a rounding difference flips one; the
        # per-sweep difference of their walker-mean energies then measures
        # the precision effect far below the runs' own statistical errors
        Kf = 4000
        cfgm = b.config()
        runs = {}
        for prec_name in (a.precision, "fp64"):
            sb = BatchedSampler([ctx], [b.walkers[0].clone()], [step], precision=prec_name,
                                proposal=a.proposal, scale_r0=HEAD_R0, scale_fmin=HEAD_FMIN,
                                cap=Kf)
            sb.configure(cfgm["threads"], cfgm["walkers_per_tile"], cfgm["variant"])
            sb.reset(EQ2 + 2 * 10**6)
            for _ in range(Kf // REFRESH_EVERY):
                sb.run(REFRESH_EVERY, 1, seed ^ 6)
            sn = sb.sums[0][:Kf].cpu().numpy()
            runs[prec_name] = (sn[:, 3] / np.maximum(sn[:, 6], 1), sb.walkers[0].clone())
            del sb
        mser, mX = runs[a.precision]
        fser, fX = runs["fp64"]
        mm, mse, _, _ = binning_analysis(mser)
        fm, fse, _, fk = binning_analysis(fser)
        dm, dse, _, _ = binning_analysis(mser - fser)
        diverged = float(torch.any((mX != fX).reshape(W, -1), dim=1).float().mean())
        ctx.set_proposal(0)
        ens = WalkerEnsemble(ctx, b.walkers[0], a.precision, seed=seed ^ 7)
        ep = torch.empty(W, 4, dtype=torch.float64, device=dev)
        ens.run(1, 1e-9, eparts_last=ep)
        ref = ctx.evaluate(ens.X, want_grad=False, want_lap=False)["e_loc"]
        dE = (ep[:, 3] - ref).cpu().numpy()
        prec = {"paired": {"sweeps": Kf, "mixed_energy": {"mean": mm, "serr": mse},
                           "fp64_energy": {"mean": fm, "serr": fse}, "fp64_tau_int": fk,
                           "diff_Ha": dm, "diff_serr_Ha": dse,
                           "walkers_diverged_frac": diverged},
                "sampled_diff_Ha": mm - fm,
                "sampled_diff_sigma": abs(mm - fm) / max(np.hypot(mse, fse), 1e-300),
                "eloc_same_configs": {"walkers": W, "mean_diff_Ha": float(dE.mean()),
                                      "serr_Ha": float(dE.std() / np.sqrt(W)),
                                      "median_abs_Ha": float(np.median(np.abs(dE))),
                                      "p99_abs_Ha": float(np.quantile(np.abs(dE), 0.99))}}
        if scaled:
            ctx.set_proposal(1, HEAD_R0, HEAD_FMIN)
        prec["outputs_vs_fp64"] = output_errors(ctx, b.walkers[0][:4096], a.precision, step,
                                                seed ^ 11)
        ctx.set_proposal(0)
        del ens

    e2e = None
    if not a.no_e2e:
        # host buffers through the public API: each call = 50 sweeps; the
        # walkers go host -> device before and device -> host after every
        # call, with the call's measurement sums
        # The copies run in E2E_CHUNKS chunks on two copy streams, so that the
        # device -> host copy of one chunk of a call's result overlaps the
        # host -> device copy of the previous chunk for the next call (the
        # two directions of the link run at once); each chunk still goes to
        # host memory and back, and every call's kernel waits for all of its
        # input
        Ke = min(n_launch, 10)
        hostX = b.walkers[0].detach().to("cpu").pin_memory()
        hsum = torch.empty(REFRESH_EVERY, NSUM, dtype=torch.float64).pin_memory()
        dX, hX = b.walkers[0].view(-1), hostX.view(-1)
        bounds = np.linspace(0, dX.numel(), E2E_CHUNKS + 1).astype(int)
        s_out, s_in = torch.cuda.Stream(), torch.cuda.Stream()
        b.reset(E2E)
        torch.cuda.synchronize()
        f0 = torch.cuda.Event(enable_timing=True)
        f1 = torch.cuda.Event(enable_timing=True)
        f0.record(stream)
        s_in.wait_stream(stream)
        with torch.cuda.stream(s_in):
            dX.copy_(hX, non_blocking=True)
        for r in range(Ke):
            stream.wait_stream(s_in)
            b.run(REFRESH_EVERY, 1, seed)
            s_out.wait_stream(stream)
            for c in range(E2E_CHUNKS):
                lo, hi = bounds[c], bounds[c + 1]
                with torch.cuda.stream(s_out):
                    hX[lo:hi].copy_(dX[lo:hi], non_blocking=True)
                    if c == E2E_CHUNKS - 1:
                        hsum.copy_(b.sums[0][r * REFRESH_EVERY:(r + 1) * REFRESH_EVERY],
                                   non_blocking=True)
                if r + 1 < Ke:
                    s_in.wait_stream(s_out)
                    with torch.cuda.stream(s_in):
                        dX[lo:hi].copy_(hX[lo:hi], non_blocking=True)
        stream.wait_stream(s_out)
        f1.record(stream)
        torch.cuda.synchronize()
        bi = b.walkers[0].numel() * 8
        e2e = {"ms_per_step": f0.elapsed_time(f1) / (Ke * REFRESH_EVERY),
               "h2d_bytes_per_step": bi / REFRESH_EVERY,
               "d2h_bytes_per_step": (bi + REFRESH_EVERY * NSUM * 8) / REFRESH_EVERY}

    t = torch.tensor([ms, e2e["ms_per_step"] if e2e else 0.0], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_max, e2e_ms = float(t[0]), float(t[1])
    wss = W * world * K / (ms_max * 1e-3)
    value = wss / kappa
    work = work_per_walker_sweep(system, acc)
    peak_kind = 0 if a.precision == "fp64" else 1
    rate = ctypes_peak(L, peak_kind)
    achieved = work["flops"] * W * REFRESH_EVERY / (launch_ms * 1e-3)
    traffic = ncu_traffic(f"{a.system}/persistent", a.precision)
    line = {
        "metric": "decorrelated samples/s (walker-steps/s / tau_int) vs plain FP64, H2O 64k walkers",
        "value": value, "unit": "decorrelated samples/s", "n_gpus": world, "steps": K,
        "steps_requested": a.steps,
        "steps_note": f"the timed region replays whole 50-sweep launches for at least "
                      f"{MIN_TIMED_S:g} s: {K} sweeps",
        "warmup": a.warmup, "ms_per_step": ms_max / K, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "f32+f64" if a.precision == "mixed" else "f64",
        "data": "synthetic",
        "config": {"workload": f"{a.system} cc-pVDZ-shaped, {W} walkers/GPU, single-electron "
                               f"sweeps + E_L every sweep, FP64 LU refresh every {REFRESH_EVERY}",
                   "precision": a.precision, "walkers_per_gpu": W, "step": step,
                   "parallelism": f"replicas x{world}",
                   "trial": "RHF determinant + Pade J2 (b=3)",
                   "kernels": "fused persistent launch per 50 sweeps (refresh, moves, E_L), "
                              f"NVRTC-specialised to the molecule (compile {t_spec:.1f} s, "
                              "untimed), CUDA graph of the timed launches",
                   "tile_shape": cfg,
                   "proposal": (f"nucleus-scaled Gaussian (r0={HEAD_R0}, fmin={HEAD_FMIN}, "
                                f"acceptance target {HEAD_ACC}), exact MH" if scaled
                                else "fixed-width Gaussian"),
                   "equilibration_sweeps": EQUIL_SWEEPS + 200,
                   "l2": "walker state in shared memory for a whole launch; positions "
                         "(15.7 MB) read and written once per 50-sweep launch"},
        "walker_sweeps_per_s": wss, "tau_int": kappa, "tau_source": tau_src,
        "energy": {"mean": e_mean, "serr": e_serr}, "acceptance": acc, "kernel_flags": flags,
        "gpu_launches": n_launch,
        "roofline": {"bound": "fp64" if peak_kind == 0 else "fp32",
                     "achieved": achieved / 1e12, "peak": rate / 1e12, "unit": "TFLOP/s",
                     "frac": achieved / rate if rate else None, "traffic": traffic,
                     "kernel": "k_batch (one launch: refresh + 50 sweeps)",
                     "kernel_ms_per_launch": launch_ms,
                     "flops_per_walker_sweep": work["flops"],
                     "flops_per_walker_sweep_dense": work["flops_dense"],
                     "mo_terms": work["mo_terms"],
                     "peak_source": "own FMA microkernel (oqmc_measure_peak), of measured"},
    }
    line["tau_int_segments"] = kq
    if plain:
        # relative uncertainty of a ratio of decorrelated rates: the two
        # kappas' standard errors (from their segments) in quadrature
        def ratio(num, k_num, s_num, den, k_den, s_den):
            r = num / den
            return {"value": r, "serr": r * float(np.hypot(s_num / k_num, s_den / k_den))}
        line["plain_fp64"] = plain
        sp = ratio(value, kappa, kq["serr"], plain["value"], plain["tau_int"],
                   plain["tau_int_segments"]["serr"])
        line["speedup_vs_plain_fp64"] = sp["value"]
        line["speedup_vs_plain_fp64_serr"] = sp["serr"]
        wk = plain["tau_int_walker_series"]
        line["speedup_vs_plain_fp64_walker_tau"] = ratio(
            value, kappa, kq["serr"], plain["walker_sweeps_per_s"] / wk["mean"], wk["mean"],
            wk["serr"])
        if fp64s:
            line["fp64_same_proposal"] = fp64s
            line["mixed_vs_fp64_same_proposal"] = ratio(
                value, kappa, kq["serr"], fp64s["value"], fp64s["tau_int"],
                fp64s["tau_int_segments"]["serr"])
            line["proposal_factor_fp64"] = ratio(
                fp64s["value"], fp64s["tau_int"], fp64s["tau_int_segments"]["serr"],
                plain["value"], plain["tau_int"], plain["tau_int_segments"]["serr"])
            line["throughput_factor_mixed_vs_fp64"] = wss / fp64s["walker_sweeps_per_s"]
    if prec:
        line["precision_check"] = prec
    if e2e:
        line["e2e"] = {"value": W * world / (e2e_ms * 1e-3) / kappa,
                       "unit": "decorrelated samples/s",
                       "h2d_bytes_per_step": e2e["h2d_bytes_per_step"],
                       "d2h_bytes_per_step": e2e["d2h_bytes_per_step"],
                       "ms_per_step": e2e_ms,
                       "note": "each API call runs 50 sweeps; walkers copied in and out per call"}
    if rank == 0 and not a.no_cpu and world == 1:
        cores = len(os.sched_getaffinity(0))
        r, kap, acc_c, sample, _ = cpu_reference(system, a.cpu_seconds, cores, (3 * 0.1) ** 0.5)
        line["cpu_baseline"] = {"value": r / kap, "unit": "decorrelated samples/s",
                                "cores": cores, "kind": "port", "sample": sample,
                                "walker_steps_per_s": r, "tau_int": kap}
    line["clocks"] = clk.summary()
    if rank == 0:
        print(json.dumps(line), flush=True)
    b.close()
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


BATCH = (("H2", 8192), ("LiH", 16384), ("H2O", 65536), ("N2", 32768), ("H2O_dimer", 16384))


def run_batched(a):
    """Five molecules of uneven size in one persistent launch per 50 sweeps,
    the launches captured in a CUDA graph, tile shape from the autotuner.

    value = walker-sweeps/s summed over the five molecules (all ranks);
    per molecule the GPU time is apportioned by the tiles' own timers."""
    import torch
    import torch.distributed as dist
    from omegaqmc_b200 import _lib as L
    from omegaqmc_b200.batch import BatchedSampler
    from omegaqmc_b200.context import GTOContext
    from omegaqmc_b200.sampler import WalkerEnsemble, init_walkers_gaussian, NSUM, PREC

    rank, world, local = dist_env()
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    names = [n for n, _ in BATCH]
    Ws = [w for _, w in BATCH]
    systems = [build_system(n) for n in names]
    ctxs, steps, X0 = [], [], []
    t_spec = time.perf_counter()
    for k, (s, W) in enumerate(zip(systems, Ws)):
        c = GTOContext(s)
        c.specialize()
        c.set_proposal(1, SCALED_R0, SCALED_FMIN)
        X = init_walkers_gaussian(s, W, 1.0, seed=100 * k + 1000 + rank)
        # step adaptation of the nucleus-scaled proposal on a 4096-walker subset
        ens = WalkerEnsemble(c, X[:4096], a.precision, seed=17 + k, refresh_every=REFRESH_EVERY)
        steps.append(a.step_size or adapt_step(ens, 0.8))
        del ens
        ctxs.append(c)
        X0.append(X)
    t_spec = time.perf_counter() - t_spec
    K = max(REFRESH_EVERY, (a.steps // REFRESH_EVERY) * REFRESH_EVERY)
    n_launch = K // REFRESH_EVERY
    b = BatchedSampler(ctxs, X0, steps, precision=a.precision, proposal="scaled",
                       scale_r0=SCALED_R0, scale_fmin=SCALED_FMIN, cap=K)
    seed = 4242 + 7919 * rank
    # equilibration (no measurements), then the autotuner, then warm-up
    # sweep-counter ranges of the phases (the RNG counter is 32-bit)
    EQ_BASE, WARM_BASE, SEP_BASE, E2E_BASE = 10**7, 2 * 10**7, 3 * 10**7, 4 * 10**7
    b.reset(EQ_BASE)
    n_eq = 0 if a.quick else EQUIL_SWEEPS // 3
    for _ in range(n_eq // REFRESH_EVERY):
        b.run(REFRESH_EVERY, REFRESH_EVERY + 1, seed)
    torch.cuda.synchronize()
    default_cfg = b.config()
    t_tune = time.perf_counter()
    cfg, tune_ms = b.tune(n_sweeps=4, seed=seed ^ 0x55)
    t_tune = time.perf_counter() - t_tune
    b.reset(WARM_BASE)
    for _ in range(max(1, a.warmup // REFRESH_EVERY)):
        b.run(REFRESH_EVERY, REFRESH_EVERY + 1, seed)
    b.capture(n_launch, REFRESH_EVERY, 1, seed)
    b.reset(0)
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    if world > 1:
        dist.barrier()
    with ClockSampler(local) as clk:
        torch.cuda.nvtx.range_push("batched_timed")
        ev0.record(stream)
        b.replay()
        ev1.record(stream)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_pop()
    ms = ev0.elapsed_time(ev1)
    busy = b.busy_ns()
    flags = b.flags()
    sums_np = [sm[:K].cpu().numpy() for sm in b.sums]

    # per-system launches of the same kernels, one after the other (the
    # comparison the batch has to beat): refresh + 50 sweeps per molecule
    sep_ms = []
    for c, X, st_, W in zip(ctxs, b.walkers, steps, Ws):
        Xc = X.clone()
        state = c.new_state(W, PREC[a.precision])
        sums = torch.zeros(REFRESH_EVERY, NSUM, dtype=torch.float64, device=dev)
        c.refresh(Xc, state, PREC[a.precision])
        c.sweeps(Xc, state, PREC[a.precision], REFRESH_EVERY, st_, seed, SEP_BASE, sums)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for r in range(2):
            c.refresh(Xc, state, PREC[a.precision])
            c.sweeps(Xc, state, PREC[a.precision], REFRESH_EVERY, st_, seed,
                     SEP_BASE + (r + 1) * REFRESH_EVERY, sums)
        e1.record(stream)
        torch.cuda.synchronize()
        sep_ms.append(e0.elapsed_time(e1) / 2)

    # e2e: walkers from pinned host memory every launch, results back
    e2e = None
    if not a.no_e2e:
        hostX = [x.detach().to("cpu").pin_memory() for x in b.walkers]
        hsums = [torch.empty(REFRESH_EVERY, NSUM, dtype=torch.float64).pin_memory()
                 for _ in b.walkers]
        Ke = min(n_launch, 10)
        b.reset(E2E_BASE)
        torch.cuda.synchronize()
        f0 = torch.cuda.Event(enable_timing=True)
        f1 = torch.cuda.Event(enable_timing=True)
        f0.record(stream)
        for r in range(Ke):
            for X, hX in zip(b.walkers, hostX):
                X.copy_(hX, non_blocking=True)
            b.run(REFRESH_EVERY, 1, seed)
            for X, hX, sm, hs in zip(b.walkers, hostX, b.sums, hsums):
                hX.copy_(X, non_blocking=True)
                hs.copy_(sm[r * REFRESH_EVERY:(r + 1) * REFRESH_EVERY], non_blocking=True)
        f1.record(stream)
        torch.cuda.synchronize()
        bi = sum(x.numel() * 8 for x in b.walkers)
        e2e = {"ms_per_step": f0.elapsed_time(f1) / (Ke * REFRESH_EVERY),
               "h2d_bytes_per_step": bi / REFRESH_EVERY,
               "d2h_bytes_per_step": (bi + len(b.walkers) * REFRESH_EVERY * NSUM * 8)
                                     / REFRESH_EVERY}
    t = torch.tensor([ms, e2e["ms_per_step"] if e2e else 0.0], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_max, e2e_ms = float(t[0]), float(t[1])

    rate = ctypes_peak(L, 0 if a.precision == "fp64" else 1)
    tot_busy = float(sum(busy))
    per = {}
    flops_total = 0.0
    dec_total = 0.0
    for k, (n, s, W) in enumerate(zip(names, systems, Ws)):
        sm = sums_np[k]
        ser = sm[:, 3] / np.maximum(sm[:, 6], 1)
        e_mean, e_serr, _, kappa = binning_analysis(ser)
        acc = float(sm[:, 5].sum() / (K * W * s.n_e))
        share = busy[k] / tot_busy
        t_k = ms * share * 1e-3
        wss = W * K / t_k
        work = work_per_walker_sweep(s, acc)
        flops_total += work["flops"] * W * K
        dec_total += W * K / (ms * 1e-3) / kappa
        per[n] = {"walkers": W, "step": steps[k], "acceptance": acc, "tau_int": kappa,
                  "energy": {"mean": e_mean, "serr": e_serr},
                  "gpu_time_share": share,
                  "walker_sweeps_per_s": wss,
                  "flops_per_walker_sweep": work["flops"],
                  "achieved_tflops": work["flops"] * W * K / t_k / 1e12,
                  "roofline_frac": work["flops"] * W * K / t_k / rate if rate else None,
                  "separate_ms_per_sweep": sep_ms[k] / REFRESH_EVERY}
    W_tot = sum(Ws)
    achieved = flops_total / (ms * 1e-3)
    line = {
        "metric": "walker-sweeps/s, H2+LiH+H2O+N2+(H2O)2 batched in one persistent launch",
        "value": W_tot * world * K / (ms_max * 1e-3), "unit": "walker-sweeps/s",
        "n_gpus": world, "steps": K, "warmup": a.warmup, "ms_per_step": ms_max / K,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32+f64" if a.precision == "mixed" else "f64", "data": "synthetic",
        "config": {"workload": "batched H2/STO-3G 8192, LiH 16384, H2O 65536, N2 32768, "
                               "(H2O)2 16384 walkers (cc-pVDZ-shaped); refresh + 50 sweeps per "
                               "launch, E_L every sweep",
                   "precision": a.precision, "parallelism": f"replicas x{world}",
                   "graph": f"{n_launch} persistent launches captured in one CUDA graph",
                   "tile_shape": cfg, "default_shape": default_cfg,
                   "autotune_s": t_tune, "compile_s": t_spec,
                   "l2": "walker state in shared memory for a whole launch; positions "
                         "(34 MB) read and written once per launch"},
        "decorrelated_samples_per_s": dec_total * world,
        "systems": per,
        "separate_launches_ms_per_sweep": sum(sep_ms) / REFRESH_EVERY,
        "batched_speedup_vs_separate": (sum(sep_ms) / REFRESH_EVERY) / (ms / K),
        "kernel_flags": flags,
        "gpu_launches": n_launch,
        "roofline": {"bound": "fp32" if a.precision == "mixed" else "fp64",
                     "achieved": achieved / 1e12, "peak": rate / 1e12 if rate else None,
                     "unit": "TFLOP/s", "frac": achieved / rate if rate else None,
                     "traffic": None, "kernel": "k_batch (generated, all five molecules)",
                     "peak_source": "own FMA microkernel (oqmc_measure_peak), of measured"},
    }
    if e2e:
        line["e2e"] = {"value": W_tot * world / (e2e_ms * 1e-3), "unit": "walker-sweeps/s",
                       "h2d_bytes_per_step": e2e["h2d_bytes_per_step"],
                       "d2h_bytes_per_step": e2e["d2h_bytes_per_step"], "ms_per_step": e2e_ms}
    line["clocks"] = clk.summary()
    if rank == 0:
        print(json.dumps(line), flush=True)
    b.close()
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


MLP_FLOPS_PER_ROW = 2 * (32 * 128 + 2 * 128 * 128 + 128 * 48)   # one forward pass


def run_learned(a):
    """N2 cc-pVDZ-shaped, 32,768 walkers, mixed precision: the plain
    fixed-width random walk against the learned MLP proposal at equal GPU
    time.  The network is trained (own tcgen05 kernels) on 10^6 walker
    configurations the plain sampler produced, targets = 8-sweep
    displacements.

    value = decorrelated samples/s of the learned sampler (walker-sweeps/s /
    tau_int of E_L); the plain sampler's figure and the ratio are reported
    beside it."""
    import torch
    import torch.distributed as dist
    from omegaqmc_b200 import _lib as L
    from omegaqmc_b200.context import GTOContext
    from omegaqmc_b200.learned import MLPProposal, collect_training_set, train_proposal
    from omegaqmc_b200.sampler import WalkerEnsemble, init_walkers_gaussian, NSUM

    rank, world, local = dist_env()
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    system = build_system("N2")
    ctx = GTOContext(system)
    ctx.specialize()
    W = 32768 if a.walkers == 65536 else a.walkers
    ens = WalkerEnsemble(ctx, init_walkers_gaussian(system, W, 1.0, seed=31 + rank), "mixed",
                         seed=2025 + 7919 * rank, refresh_every=REFRESH_EVERY)
    step = a.step_size or adapt_step(ens, STEP_DEFAULT["N2"])
    ens.run(0 if a.quick else EQUIL_SWEEPS, step)
    stream = torch.cuda.current_stream()

    def timed(e, n):
        return timed_step(e, n, step)

    def timed_step(e, n, stp):
        sums = torch.zeros(n, NSUM, dtype=torch.float64, device=dev)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        e.run(n, stp, sums=sums)
        e1.record(stream)
        torch.cuda.synchronize()
        sn = sums.cpu().numpy()
        ser = sn[:, 3] / np.maximum(sn[:, 6], 1)
        m, se, _, kap = binning_analysis(ser)
        return (e0.elapsed_time(e1), m, se, kap, float(sn[:, 5].sum() / (n * W * system.n_e)))

    # training data and training (timed with events, outside the comparison)
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    t2 = torch.cuda.Event(enable_timing=True)
    t0.record(stream)
    n_cfg = 10**5 if a.quick else 10**6
    feat, tgt = collect_training_set(ens, n_cfg, 8, step)
    t1.record(stream)
    mlp = MLPProposal(seed=11 + rank)
    n_train, batch = (300 if a.quick else 10000), 8192
    torch.cuda.nvtx.range_push("mlp_train")
    hist = train_proposal(mlp, feat, tgt, steps=n_train, batch=batch, lr=2e-3, log_every=500)
    t2.record(stream)
    torch.cuda.nvtx.range_pop()
    torch.cuda.synchronize()
    rows = int(feat.shape[0])
    del feat, tgt
    collect_ms, train_ms = t0.elapsed_time(t1), t1.elapsed_time(t2)

    # equal GPU time: the plain sampler for K_p sweeps, the learned one for
    # as many sweeps as fit in the same time
    K_p = a.steps if a.quick else max(a.steps, 1000) * 5
    ens.run(max(a.warmup, 3), step)
    with ClockSampler(local) as clk:
        ms_p, e_p, se_p, tau_p, acc_p = timed(ens, K_p)
        lens = WalkerEnsemble(ctx, ens.X, "mixed", seed=99 + rank, refresh_every=REFRESH_EVERY)
        ctx.set_mlp_proposal(mlp)
        lens.run(max(a.warmup // 10, 3), step)
        probe_ms = timed(lens, 20)[0] / 20
        K_l = max(50, int(ms_p / probe_ms))
        n_launch_l = sweep_launches(lens, K_l)
        torch.cuda.nvtx.range_push("learned_timed")
        ms_l, e_l, se_l, tau_l, acc_l = timed(lens, K_l)
        torch.cuda.nvtx.range_pop()
    flags = (ctx.flags(), mlp.flags())
    ctx.set_mlp_proposal(None)
    # the hand-built alternative at the same GPU time: the nucleus-scaled
    # Gaussian (the headline's proposal), its width adapted to acceptance 0.5
    sens = WalkerEnsemble(ctx, lens.X, "mixed", seed=77 + rank, refresh_every=REFRESH_EVERY)
    ctx.set_proposal(1, HEAD_R0, HEAD_FMIN)
    sstep = adapt_step(sens, 0.8, target=HEAD_ACC)
    sens.run(500, sstep)
    sprobe = timed_step(sens, 20, sstep)[0] / 20
    K_s = max(200, int(ms_p / sprobe))
    ms_s, e_s, se_s, tau_s, acc_s = timed_step(sens, K_s, sstep)
    ctx.set_proposal(0)
    del sens
    t = torch.tensor([ms_l, ms_p], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_l, ms_p = float(t[0]), float(t[1])
    wss_l = W * world * K_l / (ms_l * 1e-3)
    wss_p = W * world * K_p / (ms_p * 1e-3)
    value = wss_l / tau_l
    plain = wss_p / tau_p
    mlp_flops = 2.0 * system.n_e * W * K_l * MLP_FLOPS_PER_ROW
    # the driver-measured bf16 GEMM rate; without that file, the stated
    # fallback for this GPU pool (1.59 PFLOP/s)
    bf16_peak, peak_src = 1590.0, "fallback 1.59 PFLOP/s bf16 (no MEASURED_PEAKS.json), of fallback"
    peaks = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(peaks) and json.load(open(peaks)).get("bf16_tflops"):
        bf16_peak = float(json.load(open(peaks))["bf16_tflops"])
        peak_src = "MEASURED_PEAKS.json bf16_tflops, of measured"
    ach = mlp_flops / (ms_l * 1e-3) / 1e12
    train_tflops = 3.0 * n_train * batch * MLP_FLOPS_PER_ROW / (train_ms * 1e-3) / 1e12
    line = {
        "metric": "decorrelated samples/s (walker-steps/s / tau_int), learned MLP proposal vs "
                  "plain random walk at equal GPU time, N2 32k walkers",
        "value": value, "unit": "decorrelated samples/s", "n_gpus": world, "steps": K_l,
        "warmup": a.warmup, "ms_per_step": ms_l / K_l, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "bf16 (network) + f32/f64 (psi)",
        "data": "synthetic",
        "config": {"workload": f"N2 cc-pVDZ-shaped, {W} walkers/GPU, mixed precision, "
                               "single-electron sweeps + E_L every sweep",
                   "network": "per-electron MLP 32->128->128->128->48 (ReLU), 8-component "
                              "Gaussian mixture, BF16 on tcgen05",
                   "training": f"{rows} rows from {n_cfg} plain-sampler configurations "
                               f"(8-sweep displacements), {n_train} Adam steps x {batch}",
                   "equal_time": f"plain {K_p} sweeps vs learned {K_l} sweeps",
                   "parallelism": f"replicas x{world}"},
        "learned": {"tau_int": tau_l, "acceptance": acc_l, "energy": {"mean": e_l, "serr": se_l},
                    "ms_per_sweep": ms_l / K_l, "walker_sweeps_per_s": wss_l},
        "plain_random_walk": {"value": plain, "tau_int": tau_p, "acceptance": acc_p,
                              "energy": {"mean": e_p, "serr": se_p}, "step": step,
                              "ms_per_sweep": ms_p / K_p, "walker_sweeps_per_s": wss_p},
        "nucleus_scaled": {"value": W * world * K_s / (ms_s * 1e-3) / tau_s, "tau_int": tau_s,
                           "acceptance": acc_s, "energy": {"mean": e_s, "serr": se_s},
                           "step": sstep, "ms_per_sweep": ms_s / K_s, "sweeps": K_s},
        "gain_vs_scaled_equal_time": value / (W * world * K_s / (ms_s * 1e-3) / tau_s),
        "gain_equal_time": value / plain, "gain_per_sweep": tau_p / tau_l,
        "energy_diff_sigma": abs(e_l - e_p) / max(np.hypot(se_l, se_p), 1e-300),
        "training": {"collect_ms": collect_ms, "train_ms": train_ms, "loss": hist,
                     "train_tflops": train_tflops},
        "kernel_flags": list(flags),
        "gpu_launches": n_launch_l,
        "roofline": {"bound": "tensor", "achieved": ach, "peak": bf16_peak, "unit": "TFLOP/s",
                     "frac": ach / bf16_peak if bf16_peak else None, "traffic": None,
                     "kernel": "k_moves_mlp (network flops only, two passes per move)",
                     "peak_source": peak_src},
        "clocks": clk.summary(),
    }
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


def ctypes_peak(L, kind):
    import ctypes
    import torch
    lib = L.load()
    out = ctypes.c_double(0.0)
    code = lib.oqmc_measure_peak(int(kind), ctypes.byref(out),
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return out.value if code == 0 else None


def ncu_traffic(system, precision):
    """DRAM bytes per generated k_sweeps launch of 50 sweeps from the committed
    ncu summary, if any."""
    p = os.path.join(ROOT, "profiles", "ncu_traffic.json")
    if not os.path.exists(p):
        return None
    d = json.load(open(p))
    return d.get(f"{system}/{precision}")


def run_alle(a):
    """The reference's own move on the GPU: all-electron Gaussian steps with
    |psi|^2 recomputed in FP64 (oqmc_set_move_kind(ctx, 1)), the reference's
    step adaptation to acceptance 0.4, E_L every step.  One step = one
    all-electron proposal per walker.  For comparison with the single-electron
    sweeps of the headline; no roofline (a parity form, not a tuned kernel)."""
    import torch
    import torch.distributed as dist
    from omegaqmc_b200 import replicas as RP
    from omegaqmc_b200.context import GTOContext
    from omegaqmc_b200.sampler import WalkerEnsemble, init_walkers_gaussian, NSUM

    rank, world, local = dist_env()
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    system = build_system(a.system)
    ctx = GTOContext(system)
    ctx.set_move_kind(1)
    W = a.walkers
    X0 = init_walkers_gaussian(system, W, 1.0, seed=1000 + rank)
    ens = WalkerEnsemble(ctx, X0, "fp64", seed=2024 + 7919 * rank, refresh_every=REFRESH_EVERY)
    stream = torch.cuda.current_stream()
    step = a.step_size or (3 * 0.1) ** 0.5          # the reference's initial step
    if not a.quick:
        if not a.step_size:
            step = adapt_step(ens, step, n_chunks=200)
        ens.run(EQUIL_SWEEPS, step)
    ens.run(max(a.warmup, 3), step)
    K = a.steps
    sums = torch.zeros(K, NSUM, dtype=torch.float64, device=dev)
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    n_launch = fused_launches(ens, K)
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        ev0.record(stream)
        ens.run(K, step, sums=sums)
        ev1.record(stream)
        torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    t = torch.tensor([ev0.elapsed_time(ev1)], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        sums = RP.combine_sums(sums)
    ms_max = float(t[0])
    s_np = sums.cpu().numpy()
    series = s_np[:, 3] / np.maximum(s_np[:, 6], 1)
    acc = float(s_np[:, 5].sum() / (K * W * world * system.n_e))
    rate = W * world * K / (ms_max * 1e-3)
    # tau_int from a series of at least 2,000 steps: the timed one when it is
    # that long, else a separate untimed run continuing the chain
    if K >= 2000:
        tau_series, tau_src = series, f"timed series ({K} steps)"
    else:
        aux = torch.zeros(2000, NSUM, dtype=torch.float64, device=dev)
        ens.run(2000, step, sums=aux)
        if world > 1:
            aux = RP.combine_sums(aux)
        an = aux.cpu().numpy()
        tau_series = an[:, 3] / np.maximum(an[:, 6], 1)
        tau_src = "untimed 2000-step series"
    e_mean, e_serr, _, kappa = binning_analysis(tau_series)
    if rank == 0:
        print(json.dumps({
            "metric": "decorrelated samples/s, all-electron steps (the reference's move) on the GPU",
            "value": rate / kappa, "unit": "decorrelated samples/s", "n_gpus": world,
            "steps": K, "warmup": a.warmup, "ms_per_step": ms_max / K, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"{a.system} cc-pVDZ-shaped, {W} walkers/GPU, all-electron "
                                   "Gaussian steps, E_L every step, FP64",
                       "step": step, "parallelism": f"replicas x{world}"},
            "walker_steps_per_s": rate, "tau_int": kappa, "tau_source": tau_src,
            "acceptance": acc,
            "energy": {"mean": e_mean, "serr": e_serr}, "kernel_flags": ctx.flags(),
            "gpu_launches": n_launch, "roofline": None, "clocks": clk.summary()}), flush=True)
    if world > 1:
        dist.destroy_process_group()


CONFIGS = {
    # H2/STO-3G plain method: RHF, Padé J2 b = 1, 1,024 walkers from
    # N(nucleus, 0.5), fixed-width Gaussian step 0.3 bohr, 2,000 steps, FP64
    "h2": {"system": "H2", "walkers": 1024, "sigma": 0.5, "sweeps": 2000,
           "precisions": ("fp64",), "proposal": "plain", "step": 0.3, "j1": False},
    # LiH cc-pVDZ-shaped: RHF, Padé J1 (a = -Z) + J2, 16,384
    # walkers from N(nucleus, 1.0); FP64 against mixed with the same proposal
    "lih": {"system": "LiH", "walkers": 16384, "sigma": 1.0, "sweeps": 2000,
            "precisions": ("mixed", "fp64"), "proposal": "scaled", "step": 0.0, "j1": True},
}


def run_config(a):
    """The H2/STO-3G and LiH workloads through the persistent path: per
    precision, equilibration, then whole 50-sweep launches replayed from a
    CUDA graph for the workload's sweep count (repeated until at least
    1 s is timed); tau_int from the timed series.  LiH adds the error of
    every per-walker output of the mixed sampler against the FP64
    evaluation on 4,096 fixed seeded configurations."""
    import torch
    from omegaqmc_b200 import _lib as L  # noqa: F401
    from omegaqmc_b200 import molecules as M
    from omegaqmc_b200.batch import BatchedSampler
    from omegaqmc_b200.context import GTOContext
    from omegaqmc_b200.sampler import init_walkers_gaussian
    from omegaqmc_b200.system import build_system as bs

    rank, world, local = dist_env()
    if rank != 0:
        return
    cf = CONFIGS[a.workload]
    torch.cuda.set_device(local)
    mf = M.make_mf(cf["system"])
    system = bs(mf, M.default_params_corr(mf.mol, j1=cf["j1"]))
    ctx = GTOContext(system)
    ctx.specialize()
    W, Kc = cf["walkers"], cf["sweeps"]
    X0 = init_walkers_gaussian(system, W, cf["sigma"], seed=77)
    stream = torch.cuda.current_stream()
    arms = {}
    launches = 0
    clk_summary = None
    for prec in cf["precisions"]:
        b = BatchedSampler([ctx], [X0], [cf["step"] or 0.8], precision=prec,
                           proposal=cf["proposal"], scale_r0=HEAD_R0, scale_fmin=HEAD_FMIN,
                           cap=Kc)
        if not cf["step"]:
            b.adapt_steps(HEAD_ACC, seed=5)
        b.reset(10**7)
        for _ in range(max(a.warmup, 3) + 20):
            b.run(REFRESH_EVERY, REFRESH_EVERY + 1, 9)
        cfg, _ = b.tune(4, seed=6)
        n_l = Kc // REFRESH_EVERY
        b.capture(n_l, REFRESH_EVERY, 1, 9)
        reps, total_ms, series = 0, 0.0, None
        with ClockSampler(local) as clk:
            while reps == 0 or (total_ms < 1000.0 and reps < 200):
                b.reset(reps * Kc)
                torch.cuda.synchronize()
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                b.replay()
                e1.record(stream)
                torch.cuda.synchronize()
                total_ms += e0.elapsed_time(e1)
                reps += 1
                if series is None:
                    sn = b.sums[0][:Kc].cpu().numpy()
                    series = sn[:, 3] / np.maximum(sn[:, 6], 1)
                    acc = float(sn[:, 5].sum() / (Kc * W * system.n_e))
        launches += reps * n_l
        clk_summary = clk.summary()
        mean, serr, _, kappa = binning_analysis(series)
        wss = W * Kc * reps / (total_ms * 1e-3)
        arms[prec] = {"value": wss / kappa, "walker_sweeps_per_s": wss, "tau_int": kappa,
                      "ms_per_step": total_ms / (Kc * reps), "timed_repeats": reps,
                      "step": b.steps()[0], "acceptance": acc, "tile_shape": cfg,
                      "energy": {"mean": mean, "serr": serr}, "kernel_flags": b.flags()}
        b.close()
        del b
    main_prec = cf["precisions"][0]
    m = arms[main_prec]
    line = {
        "metric": f"decorrelated samples/s (walker-steps/s / tau_int), {cf['system']} "
                  f"{W} walkers",
        "value": m["value"], "unit": "decorrelated samples/s", "n_gpus": 1, "steps": Kc,
        "warmup": a.warmup, "ms_per_step": m["ms_per_step"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if main_prec == "fp64" else "f32+f64", "data": "synthetic",
        "config": {"workload": f"{a.workload}: {cf['system']} "
                               f"{'STO-3G' if cf['system'] == 'H2' else 'cc-pVDZ-shaped'}, "
                               f"RHF, Pade {'J1+J2' if cf['j1'] else 'J2'} (b=1), {W} walkers "
                               f"from N(nucleus, {cf['sigma']}), {Kc} single-electron sweeps "
                               "with E_L every sweep per timed repeat",
                   "proposal": ("fixed-width Gaussian" if cf["proposal"] == "plain" else
                                f"nucleus-scaled Gaussian (r0={HEAD_R0}, fmin={HEAD_FMIN})"),
                   "precision": main_prec},
        "tau_int": m["tau_int"], "energy": m["energy"], "acceptance": m["acceptance"],
        "walker_sweeps_per_s": m["walker_sweeps_per_s"], "arms": arms,
        "gpu_launches": launches, "roofline": None, "clocks": clk_summary}
    if "fp64" in arms and main_prec != "fp64":
        f = arms["fp64"]
        line["mixed_vs_fp64"] = m["value"] / f["value"]
        line["energy_diff_sigma"] = abs(m["energy"]["mean"] - f["energy"]["mean"]) / max(
            np.hypot(m["energy"]["serr"], f["energy"]["serr"]), 1e-300)
        Xf = torch.tensor(init_walkers_gaussian(system, 4096, cf["sigma"], seed=2024),
                          dtype=torch.float64, device="cuda")
        ctx.set_proposal(1, HEAD_R0, HEAD_FMIN)
        line["outputs_vs_fp64"] = output_errors(ctx, Xf, main_prec, m["step"], 11)
        ctx.set_proposal(0)
    if not a.no_cpu:
        cores = len(os.sched_getaffinity(0))
        r, kap, acc_c, sample, ser = cpu_reference(system, a.cpu_seconds, cores,
                                                   cf["step"] or (3 * 0.1) ** 0.5)
        cm, cse, _, _ = binning_analysis(ser)
        line["cpu_baseline"] = {"value": r / kap, "unit": "decorrelated samples/s",
                                "cores": cores, "kind": "port", "sample": sample,
                                "walker_steps_per_s": r, "tau_int": kap,
                                "energy": {"mean": cm, "serr": cse}}
        line["energy_vs_cpu_reference_sigma"] = abs(m["energy"]["mean"] - cm) / max(
            np.hypot(m["energy"]["serr"], cse), 1e-300)
    print(json.dumps(line), flush=True)


def main():
    a = parse()
    if a.impl == "reference":
        run_reference(a)
    elif a.workload == "alle":
        run_alle(a)
    elif a.workload in CONFIGS:
        run_config(a)
    elif a.workload == "batched":
        run_batched(a)
    elif a.workload == "learned":
        run_learned(a)
    elif a.path == "split" or a.eloc == "tc":
        run_ours(a)
    else:
        run_persistent(a)


if __name__ == "__main__":
    main()
