"""Fused sweeps with several lanes per walker: every lane count the walker
count can select (and walkers that leave a warp or a tile partly empty)
against the same sweeps with one lane per walker, which a CTA size asked for
by the caller selects, and the last local energies against the oracle.

Mixed precision: the lanes keep the one-lane order of every FP32 sum, so the
walkers are identical.  FP64: the pair sums are added in another order
(relative 1e-15), which parts two chains only where an acceptance lies that
close to its uniform, so at most one walker of 10^4 may differ."""
import numpy as np
import pytest
import torch

from helpers import seeded_walkers
from oracle import gto_oracle as O
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.context import GTOContext
from omegaqmc_b200.sampler import WalkerEnsemble
from omegaqmc_b200.system import build_system

pytestmark = pytest.mark.gpu


def _system(name, j3):
    mol = M.named_system(name)
    pc = M.default_params_corr(mol)
    cfg = None
    if j3:
        n = {2: 8, 3: 26}[j3]
        rng = np.random.default_rng(4)
        pc["J3_eeI"] = {p + e: rng.normal(size=n) * 0.003 for e in sorted(set(mol.elements))
                        for p in ("like+", "unlike+") if p + e != "like+H"}
        cfg = {"J3": {"N_eI": j3, "N_ee": j3, "r_cut": 4.0}}
    return build_system(M.make_mf(name), pc, None, cfg)


# H2O, 10 electrons: 16, 8, 4, 2 lanes; LiH: 4, 2; H2: 2; the dimer: 32;
# three-body terms: 32 and 16
CASES = [("H2O", "fp64", 37, 0, 1, 0), ("H2O", "mixed", 37, 0, 0, 0),
         ("H2O", "fp64", 5003, 0, 1, 0), ("H2O", "mixed", 12001, 0, 1, 0),
         ("H2O", "fp64", 20001, 0, 0, 0), ("LiH", "mixed", 33, 0, 1, 0),
         ("LiH", "fp64", 20001, 0, 1, 0), ("H2", "fp64", 65, 0, 0, 0),
         ("H2O_dimer", "fp64", 9, 0, 1, 0), ("H2O", "fp64", 17, 2, 0, 0),
         ("H2O", "fp64", 3001, 3, 1, 0), ("LiH", "mixed", 129, 2, 0, 0),
         ("H2O", "fp64", 101, 0, 1, 1), ("LiH", "mixed", 300, 0, 1, 1)]


@pytest.mark.parametrize("name,prec,W,j3,prop,spec", CASES)
def test_lanes_follow_one_lane(name, prec, W, j3, prop, spec):
    s = _system(name, j3)
    ctx = GTOContext(s)
    if spec:
        ctx.specialize()
    ctx.set_proposal(prop)
    X = seeded_walkers(s, W, 0.9, 31)
    n, every = 7, 2                       # three measurements and a sweep after them
    out = []
    for wpb in (32, 0):
        ens = WalkerEnsemble(ctx, X, prec, seed=9, refresh_every=10**9, walkers_per_block=wpb)
        ep = torch.zeros(W, 4, dtype=torch.float64, device="cuda")
        tr = torch.zeros(n // every, W, dtype=torch.float64, device="cuda")
        sums = ens.run(n - 1, 0.4, measure_every=every, eparts_last=ep, el_trace=tr)
        Xm = ens.X.clone()
        ens.run(1, 0.4)
        st = ens.state_evaluate()
        out.append((Xm, ens.X, sums, ep, tr, st["logpsi"], st["e_loc"]))
    a, b = out
    same = torch.all((a[1] == b[1]).view(W, -1), dim=1)
    if prec == "mixed":
        assert bool(same.all())
    else:
        assert int((~same).sum()) <= W // 10000
    assert not torch.equal(b[0], b[1])
    # sums over walkers: FP64 additions in another order
    assert torch.allclose(a[2][:, 5:], b[2][:, 5:], rtol=2e-4)
    if bool(same.all()):
        tol = 1e-9 if prec == "fp64" else 1e-12
        assert torch.allclose(a[2][:, :5], b[2][:, :5], rtol=tol)
        assert torch.allclose(a[5], b[5], rtol=1e-10, atol=1e-10)
    # the last measurement against the oracle at its walkers
    m = min(W, 200)
    o = O.evaluate(s, b[0][:m].cpu().numpy())
    sc = 0.5 * (np.sum(np.abs(o["lap"]), axis=1) + np.sum(o["grad"] ** 2, axis=(1, 2))) + 1.0
    ep = b[3][:m].cpu().numpy()
    tol = 1e-9 if prec == "fp64" else 2e-3
    assert np.max(np.abs(ep[:, 3] - o["e_loc"]) / (np.abs(o["e_loc"]) + sc)) < tol
    assert torch.equal(b[4][-1], b[3][:, 3])
    assert ctx.flags() == 0


@pytest.mark.parametrize("name,prec,W", [("H2O", "fp64", 45), ("LiH", "mixed", 9000),
                                         ("H2", "fp64", 70000)])
def test_device_adaptation_counts_every_walker(name, prec, W):
    """The last CTA of an equilibration step adapts the width from the exact
    number of accepted moves of all CTAs: the recorded ratios are whole
    multiples of 1 / (W n_e) and follow the width rule."""
    s = _system(name, 0)
    ctx = GTOContext(s)
    ens = WalkerEnsemble(ctx, seeded_walkers(s, W, 0.9, 3), prec, seed=2, refresh_every=3)
    step, acc, widths = ens.equilibrate(8, 0.5, target=0.4, rate=0.05)
    acc, widths = acc.cpu().numpy(), widths.cpu().numpy()
    n = acc * W * s.n_e
    assert np.max(np.abs(n - np.round(n))) < 1e-6 and np.all((n > 0) & (n <= W * s.n_e))
    w = np.concatenate([[0.5], widths])
    np.testing.assert_allclose(w[1:], w[:-1] * np.exp(0.05 * (acc - 0.4)), rtol=1e-13)
    assert step == widths[-1]
    ens2 = WalkerEnsemble(ctx, seeded_walkers(s, W, 0.9, 3), prec, seed=2, refresh_every=3)
    for k in range(8):
        ens2.run(1, float(w[k]))
    assert torch.equal(ens.X, ens2.X)
