"""Performance cases of the framework: what its users have it do, through its public entry points.

Every case names a path (``kind``), a molecule of :data:`omegaqmc_b200.molecules.NAMED_SYSTEMS`
and its sizes.  The paths:

``evaluate``  ``GTOContext.evaluate``: log|psi|, its gradient and Laplacians and the local energy
              of given walkers (the wavefunction surface behind ``get_psi_fun``), FP64
``logpsi``    ``GTOContext.log_psi``: the value path, FP64
``derivs``    ``optim.walker_derivatives``: the linear-method optimiser's inputs per walker
``sweeps``    ``WalkerEnsemble.run``: single-electron sweeps with a local energy after each
``equil``     ``WalkerEnsemble.equilibrate``: sweeps with the step width adapted after each
``alle``      ``WalkerEnsemble.run`` with the reference's all-electron step
``batch``     ``BatchedSampler.run``: the fused persistent launch of the driver's production blocks
``train``     ``MLPProposal.backward``: the learned proposal's loss and gradient on the tensor cores

Contexts, samplers and networks do not depend on the walkers, so they are made once per process,
as a program keeps them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from omegaqmc_b200 import molecules as M
from omegaqmc_b200.batch import BatchedSampler
from omegaqmc_b200.context import GTOContext
from omegaqmc_b200.learned import MLPProposal
from omegaqmc_b200.optim import walker_derivatives
from omegaqmc_b200.sampler import WalkerEnsemble
from omegaqmc_b200.system import build_system

DEV = "cuda"
_HANDLES = {}


def listed():
    return [
        # one walker: an interactive call or a test, where only latency counts
        {"name": "evaluate_h2o_1", "kind": "evaluate", "mol": "H2O", "walkers": 1},
        # the size the parity tests evaluate, one more than a multiple of every tile
        {"name": "evaluate_n2_4097", "kind": "evaluate", "mol": "N2", "walkers": 4097},
        # the largest named molecule with a production walker count
        {"name": "evaluate_dimer_16384", "kind": "evaluate", "mol": "H2O_dimer",
         "walkers": 16384},
        # the benchmark's walkers through the value path (checking a walker set, reweighting)
        {"name": "logpsi_h2o_65536", "kind": "logpsi", "mol": "H2O", "walkers": 65536},
        # one optimiser iteration's sample with a three-body Jastrow
        {"name": "derivs_h2o_j3_2048", "kind": "derivs", "mol": "H2O", "walkers": 2048,
         "j3": True},
        # the benchmark's smallest workload: H2/STO-3G, 1,024 walkers, plain FP64 sampler
        {"name": "sweeps_h2_1024", "kind": "sweeps", "mol": "H2", "walkers": 1024, "sweeps": 50,
         "precision": "fp64", "proposal": 0, "j3": False},
        # sampling with the three-body Jastrow (an optimiser's sampling stage)
        {"name": "sweeps_h2o_j3_2048", "kind": "sweeps", "mol": "H2O", "walkers": 2048,
         "sweeps": 20, "precision": "fp64", "proposal": 0, "j3": True},
        # the benchmark's LiH workload: mixed precision, nucleus-scaled proposal
        {"name": "sweeps_lih_16384", "kind": "sweeps", "mol": "LiH", "walkers": 16384,
         "sweeps": 50, "precision": "mixed", "proposal": 1, "j3": False},
        # the driver's defaults: 1,000 walkers, one block of 100 equilibration steps
        {"name": "equil_h2o_1000", "kind": "equil", "mol": "H2O", "walkers": 1000,
         "sweeps": 100},
        # the reference's own move, every electron at once
        {"name": "alle_h2o_16384", "kind": "alle", "mol": "H2O", "walkers": 16384, "sweeps": 10},
        # the headline: H2O, 65,536 walkers, 50 sweeps per launch, local energy every sweep
        {"name": "batch_h2o_65536", "kind": "batch", "mol": "H2O", "walkers": 65536,
         "sweeps": 50},
        # one training batch of the learned proposal
        {"name": "train_8192", "kind": "train", "rows": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "logpsi", "derivs", "sweeps", "equil", "alle", "batch",
                       "train", "evaluate", "sweeps"])
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 500, 8192)}
    if kind in ("evaluate", "logpsi"):
        mol = rng.choice(["H2", "LiH", "H2O", "N2", "H2O_dimer"])
        hi = 65536 if kind == "logpsi" else 16384
        return {"kind": kind, "mol": mol, "walkers": _log_int(rng, 1, hi)}
    if kind == "derivs":
        return {"kind": kind, "mol": rng.choice(["LiH", "H2O"]),
                "walkers": _log_int(rng, 100, 2048), "j3": rng.random() < 0.7}
    if kind == "sweeps":
        mixed = rng.random() < 0.4
        return {"kind": kind, "mol": rng.choice(["H2", "LiH", "H2O"]),
                "walkers": _log_int(rng, 1000, 16384) if mixed else _log_int(rng, 200, 4096),
                "sweeps": rng.randint(5, 50), "precision": "mixed" if mixed else "fp64",
                "proposal": 1 if mixed else rng.randint(0, 1),
                "j3": not mixed and rng.random() < 0.3}
    if kind == "equil":
        return {"kind": kind, "mol": rng.choice(["H2", "LiH", "H2O"]),
                "walkers": _log_int(rng, 200, 4096), "sweeps": rng.randint(20, 100)}
    if kind == "alle":
        return {"kind": kind, "mol": rng.choice(["H2", "LiH", "H2O"]),
                "walkers": _log_int(rng, 200, 16384), "sweeps": rng.randint(2, 20)}
    return {"kind": kind, "mol": rng.choice(["LiH", "H2O"]),
            "walkers": _log_int(rng, 4096, 65536), "sweeps": rng.randint(10, 50)}


# -- handles --------------------------------------------------------------------------------------
def _j3_params(mol):
    """Free parameters of a three-body Jastrow (orders 2 and 2) per element, of the size the
    tests use."""
    g = np.random.default_rng(5)
    els = sorted(set(mol.elements))
    return {p + e: g.normal(size=8) * 0.004 for e in els for p in ("like+", "unlike+")
            if p + e != "like+H"}


def _params(case):
    mol = M.named_system(case["mol"])
    if case["kind"] in ("evaluate", "logpsi", "derivs") or case.get("j3"):
        pc = M.default_params_corr(mol)
    else:
        pc = M.benchmark_params_corr(mol)
    cfg = None
    if case.get("j3"):
        pc["J3_eeI"] = _j3_params(mol)
        cfg = {"J3": {"N_eI": 2, "N_ee": 2, "r_cut": 4.0}}
    return pc, cfg


def _system(case):
    key = ("system", case["mol"], case["kind"] in ("evaluate", "logpsi", "derivs"),
           bool(case.get("j3")))
    if key not in _HANDLES:
        pc, cfg = _params(case)
        _HANDLES[key] = build_system(M.make_mf(case["mol"]), pc, None, cfg)
    return _HANDLES[key]


def _context(case):
    sampling = case["kind"] in ("sweeps", "equil", "batch")
    move = 1 if case["kind"] == "alle" else 0
    key = ("context", case["mol"], case["kind"] in ("evaluate", "logpsi", "derivs"),
           bool(case.get("j3")), sampling, move, case.get("proposal", 0))
    if key not in _HANDLES:
        ctx = GTOContext(_system(case))
        if sampling and case["kind"] != "batch":
            ctx.specialize()                       # as the driver does
        if case.get("proposal"):
            ctx.set_proposal(1, 1.0, 0.05)
        ctx.set_move_kind(move)
        _HANDLES[key] = ctx
    return _HANDLES[key]


def _walkers(case, seed):
    """(W, n_e, 3) electrons N(nucleus, 1 bohr), assigned to nuclei by charge: the benchmark's
    initial state."""
    s = _system(case)
    idx = np.repeat(np.arange(s.natm), s.Z.astype(int))[: s.n_e]
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & (2**63 - 1))
    x = torch.randn(case["walkers"], s.n_e, 3, generator=g, device=DEV, dtype=torch.float64)
    return x + torch.as_tensor(s.nuc[idx], device=DEV)


STEP = {"H2": 0.3, "LiH": 0.3, "H2O": 0.3}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        if "mlp" not in _HANDLES:
            _HANDLES["mlp"] = MLPProposal(seed=3)
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed) & (2**63 - 1))
        feat = torch.randn(case["rows"], 32, generator=g, device=DEV).bfloat16()
        feat[:, 31] = 1.0
        tgt = 0.3 * torch.randn(case["rows"], 3, generator=g, device=DEV)
        return {"case": case, "mlp": _HANDLES["mlp"], "feat": feat.view(torch.int16),
                "target": tgt}
    ctx = _context(case)
    X = _walkers(case, seed)
    st = {"case": case, "ctx": ctx, "X": X, "seed": int(seed) & 0x7FFFFFFF}
    if kind in ("sweeps", "equil", "alle"):
        st["ens"] = WalkerEnsemble(ctx, X, case.get("precision", "fp64"), seed=st["seed"])
    if kind == "derivs":
        st["params"] = _params(case)[0]
    if kind == "batch":
        key = ("batch", case["mol"], case["walkers"], case["sweeps"])
        if key not in _HANDLES:
            b = BatchedSampler([ctx], [X.clone()], [STEP[case["mol"]]], precision="mixed",
                               proposal="scaled", cap=case["sweeps"])
            b.configure(64, [64], 2)               # the shape the autotuner picks for H2O
            _HANDLES[key] = b
        st["batch"] = _HANDLES[key]
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "evaluate":
        return st["ctx"].evaluate(st["X"])
    if kind == "logpsi":
        return st["ctx"].log_psi(st["X"])
    if kind == "derivs":
        return walker_derivatives(st["ctx"], st["X"], st["params"])
    if kind == "train":
        grad, loss = st["mlp"].backward(st["feat"], st["target"])
        return {"grad": grad, "loss": loss}
    if kind == "sweeps":
        sums = st["ens"].run(case["sweeps"], STEP[case["mol"]])
        # the mixed build's energies are FP32 arithmetic summed in FP64
        return {"walkers": st["ens"].X,
                "sums": sums.float() if case["precision"] == "mixed" else sums}
    if kind == "equil":
        step, acc, widths = st["ens"].equilibrate(case["sweeps"], STEP[case["mol"]])
        return {"walkers": st["ens"].X, "step": step, "acceptance": acc, "widths": widths}
    if kind == "alle":
        sums = st["ens"].run(case["sweeps"], 0.08)
        return {"walkers": st["ens"].X, "sums": sums}
    b = st["batch"]                                # walkers in, one launch, walkers out
    b.walkers[0].copy_(st["X"])
    b.reset(0)
    b.run(case["sweeps"], 1, st["seed"])
    st["X"].copy_(b.walkers[0])
    return {"walkers": st["X"], "sums": b.sums[0][: case["sweeps"]].float()}


# -- what a pass cannot do without ----------------------------------------------------------------
def _counts(case):
    """(electrons, orbitals per spin, basis functions, primitives, nuclei) of the molecule."""
    s = _system(case)
    nprim = sum(len(a) for _, a, _ in s.prim_groups())
    return s.n_e, s.nocc, s.nbf, nprim, s.natm


def work(case):
    if case["kind"] == "train":
        return {"bytes": case["rows"] * (64 + 12) + 43440 * 12,
                "flops": 3 * 83968.0 * case["rows"]}
    ne, no, nbf, npr, nat = _counts(case)
    W = case["walkers"]
    pairs = ne * (ne - 1) / 2 + ne * nat
    exp, inv = 20.0, 2 * (2.0 * no ** 3)           # flops of one exponential, both inverses
    value = ne * (npr * (exp + 4) + 2 * nbf * no) + 15 * pairs
    vgl = ne * (npr * (exp + 12) + 10 * nbf * no) + 40 * pairs
    x = 8.0 * W * 3 * ne
    if case["kind"] == "logpsi":
        return {"bytes": x + 8.0 * W, "flops": W * (value + inv)}
    if case["kind"] == "evaluate":
        return {"bytes": 2 * x + 8.0 * W * (ne + 5), "flops": W * (vgl + inv)}
    if case["kind"] == "derivs":
        npar = 5 + 24 * bool(case["j3"])
        j3 = 18 * 60.0 * pairs * bool(case["j3"])
        return {"bytes": x + 8.0 * W * (1 + 2 * npar), "flops": W * (vgl + inv + j3)}
    # contracted with the inverse column first, the local energy needs ~4 terms per coefficient
    move = ne * (npr * (exp + 4) + 2 * nbf * no + 6 * no * no + 60) + 30 * 2 * pairs
    local = ne * (npr * (exp + 12) + 8 * nbf * no) + 40 * pairs
    if case.get("j3"):
        move += 2 * 40.0 * pairs * nat
        local += 120.0 * pairs * nat
    if case["kind"] == "alle":
        move = value + inv
    if case["kind"] == "equil":
        local = 0.0
    return {"bytes": 2 * x + 64.0 * case["sweeps"], "flops": W * case["sweeps"] * (move + local)}


# -- the same in plain 64-bit torch ---------------------------------------------------------------
def _harmonics(am, d):
    """Real solid harmonics of a displacement (..., 3) and their gradients (..., 2 am + 1, 3)."""
    x, y, z = d.unbind(-1)
    o, zero = torch.ones_like(x), torch.zeros_like(x)
    if am == 0:
        return o[..., None], torch.zeros_like(d)[..., None, :]
    if am == 1:
        return d, torch.eye(3, dtype=d.dtype, device=d.device).expand(*d.shape, 3)
    if am != 2:
        raise ValueError(am)
    c, h = math.sqrt(3.0), math.sqrt(3.0) / 2
    Y = [c * x * y, c * y * z, z * z - 0.5 * (x * x + y * y), c * x * z, h * (x * x - y * y)]
    G = [[c * y, c * x, zero], [zero, c * z, c * y], [-x, -y, 2 * z], [c * z, zero, c * x],
         [c * x, -c * y, zero]]
    return torch.stack(Y, -1), torch.stack([torch.stack(g, -1) for g in G], -2)


def _exact_chunk(s, X):
    """log|psi|, gradient, Laplacians and energies of walkers X in 64 bits: Slater determinants
    of the molecular orbitals and Padé Jastrow terms."""
    T = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=X.device)  # noqa: E731
    W, ne, _ = X.shape
    C, nuc, Z = T(s.C), T(s.nuc), T(s.Z)
    chi, dchi, lchi = [], [], []
    for sh in s.shells:
        d = X - nuc[sh.iat]
        r2 = (d * d).sum(-1)
        a, n = T(sh.alpha), T(sh.norm)
        e = torch.exp(-a * r2[..., None]) * n
        R, R1, R2 = e.sum(-1), (-a * e).sum(-1), (a * a * e).sum(-1)      # in s = r^2
        Y, dY = _harmonics(sh.am, d)
        chi.append(R[..., None] * Y)
        dchi.append(2 * (R1[..., None] * Y)[..., None] * d[..., None, :] + R[..., None, None] * dY)
        lchi.append((4 * r2 * R2 + (6 + 4 * sh.am) * R1)[..., None] * Y)
    phi = torch.cat(chi, -1) @ C
    dphi = torch.einsum("weac,am->wemc", torch.cat(dchi, -2), C)
    lphi = torch.cat(lchi, -1) @ C
    logpsi = torch.zeros(W, dtype=X.dtype, device=X.device)
    grad, lap = torch.zeros_like(X), torch.zeros_like(X[..., 0])
    for sp in (0, 1):
        S = phi[:, sp::2]
        logpsi = logpsi + torch.linalg.slogdet(S)[1]
        A = torch.linalg.inv(S)
        g = torch.einsum("wmi,wimc->wic", A, dphi[:, sp::2])
        grad[:, sp::2] = g
        lap[:, sp::2] = torch.einsum("wmi,wim->wi", A, lphi[:, sp::2]) - (g * g).sum(-1)

    def pade(a, b, d, r):
        q = 1 / (1 + b * r)
        return a * r * q, (a * q * q / r)[..., None] * d, -2 * a * b * q ** 3 + 2 * a * q * q / r

    e_ee = torch.zeros_like(logpsi)
    e_en = torch.zeros_like(logpsi)
    for i in range(ne):
        for j in range(i + 1, ne):
            d = X[:, i] - X[:, j]
            r = d.norm(dim=-1)
            e_ee = e_ee + 1 / r
            if s.has_j2:
                a, b = [float(v) for v in np.ravel(s.j2)[(0 if (i - j) % 2 == 0 else 2):][:2]]
                u, g, l = pade(a, b, d, r)
                logpsi = logpsi + u
                grad[:, i] += g
                grad[:, j] -= g
                lap[:, i] += l
                lap[:, j] += l
        for k in range(len(Z)):
            d = X[:, i] - nuc[k]
            r = d.norm(dim=-1)
            e_en = e_en - Z[k] / r
            if s.has_j1:
                a, b = [float(v) for v in np.reshape(s.j1, (len(Z), -1))[k][:2]]
                u, g, l = pade(a, b, d, r)
                logpsi = logpsi + u
                grad[:, i] += g
                lap[:, i] += l
    ke = -0.5 * (lap.sum(1) + (grad * grad).sum((1, 2)))
    return {"logpsi": logpsi, "e_ee": e_ee, "e_en": e_en, "e_ke": ke,
            "e_loc": e_ee + e_en + ke + float(s.e_nn), "grad": grad, "lap": lap}


def _exact_train(case, seed):
    st = prepare(case, seed)
    th = torch.as_tensor(st["mlp"].params().astype(np.float64), device=DEV).requires_grad_(True)
    h, o = st["feat"].view(torch.bfloat16).double(), 0
    for n, k in ((128, 32), (128, 128), (128, 128), (48, 128)):
        w, b = th[o:o + n * k].view(n, k), th[o + n * k:o + n * k + n]
        o += n * k + n
        h = h @ w.T + b
        h = torch.relu(h) if n == 128 else h
    mu = h[:, 8:32].view(-1, 8, 3)
    sig = 0.02 + torch.nn.functional.softplus(h[:, 32:40])
    r2 = ((st["target"].double()[:, None, :] - mu) ** 2).sum(-1)
    lq = torch.logsumexp(torch.log_softmax(h[:, :8], 1) - 3 * torch.log(sig)
                         - 1.5 * math.log(2 * math.pi) - 0.5 * r2 / sig ** 2, 1)
    loss = -lq.mean()
    loss.backward()
    return {"grad": th.grad, "loss": loss.detach()}


def exact(case, seed):
    """Evaluations and training gradients; a Markov chain has no value of its own to compare."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] not in ("evaluate", "logpsi"):
        return None
    s, X = _system(case), _walkers(case, seed)
    parts = [_exact_chunk(s, x) for x in X.split(4096)]
    out = {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    return out["logpsi"] if case["kind"] == "logpsi" else out
