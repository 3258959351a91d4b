"""The sweeps of one thread per walker: above the walker counts that lanes
serve, systems without compiled-in orbitals or with three-body terms move in
k_moves and take their local energies from k_eloc, as do FP64 ensembles of
eight and more orbitals, and FP64 ones whose caller asks for small CTAs.  The
local energies are then the ones that state_evaluate forms with the same
kernel, bit for bit, and the chains are those of smaller ensembles, whose
walkers share lanes."""
import numpy as np
import pytest
import torch

from helpers import golden_system, seeded_walkers
from oracle import gto_oracle as O
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.context import GTOContext
from omegaqmc_b200.sampler import WalkerEnsemble
from omegaqmc_b200.system import build_system

pytestmark = pytest.mark.gpu


def _system(name):
    if name.startswith("golden:"):
        return golden_system(name[7:])[0]
    mol = M.named_system(name.split("+")[0])
    pc, cfg = M.default_params_corr(mol), None
    if "+j" in name:
        k = 3 if name.endswith("j33") else 2
        rng = np.random.default_rng(4)
        pc["J3_eeI"] = {p + e: rng.normal(size={2: 8, 3: 26}[k]) * 0.003
                        for e in sorted(set(mol.elements))
                        for p in ("like+", "unlike+") if p + e != "like+H"}
        cfg = {"J3": {"N_eI": k, "N_ee": k, "r_cut": 4.0}}
    return build_system(M.make_mf(name.split("+")[0]), pc, None, cfg)


def _ensemble(ctx, s, W, prec, wpb=0):
    X = seeded_walkers(s, 512, 0.9, 31)
    return WalkerEnsemble(ctx, np.tile(X, (-(-W // 512), 1, 1))[:W], prec, seed=9,
                          refresh_every=10**9, walkers_per_block=wpb)


# just above the counts at which the last lanes are given up (37,888 = 148 x 512 / 2;
# 28,416 where three CTAs of two lanes no longer hold all walkers at once;
# three-body terms in FP32: 148 x 256 / 16 = 2,368, 148 x 128 / 16 = 1,184 and
# 148 x 256 / 4 = 9,472), with a partial last CTA
CASES = [("H2O", "mixed", 37889, 0, 0, 0), ("H2O", "fp64", 37889, 0, 1, 0),
         ("golden:h2o_cusp", "mixed", 40001, 0, 0, 0), ("H2O+j3", "mixed", 2369, 1, 0, 0),
         ("H2O+j3", "mixed", 2369, 1, 1, 0), ("H2O+j33", "mixed", 1185, 0, 0, 0),
         ("H2O", "fp64", 28417, 0, 0, 0), ("N2", "mixed", 28417, 0, 1, 0),
         ("LiH+j3", "mixed", 9473, 1, 1, 0), ("LiH+j3", "fp64", 37889, 1, 0, 0),
         ("H2O+j3", "fp64", 37889, 1, 0, 0), ("H2O_dimer", "fp64", 37889, 1, 0, 0),
         ("H2O", "fp64", 1001, 1, 0, 32), ("H2O", "fp64", 1001, 1, 1, 128)]


@pytest.mark.parametrize("name,prec,W,spec,prop,wpb", CASES)
def test_one_thread_per_walker(name, prec, W, spec, prop, wpb):
    s = _system(name)
    ctx = GTOContext(s)
    if spec:
        ctx.specialize()
    ctx.set_proposal(prop)
    ens = _ensemble(ctx, s, W, prec, wpb)
    ep = torch.zeros(W, 4, dtype=torch.float64, device="cuda")
    tr = torch.zeros(3, W, dtype=torch.float64, device="cuda")
    sums = ens.run(6, 0.4, measure_every=2, eparts_last=ep, el_trace=tr)
    assert torch.equal(tr[-1], ep[:, 3])
    assert bool((sums[:, 6] == W).all()) and abs(float(sums[-1, 3] - ep[:, 3].sum())) < 1e-9 * float(
        ep[:, 3].abs().sum())
    st = ens.state_evaluate()
    for k, q in enumerate(("e_ee", "e_en", "e_ke", "e_loc")):
        assert torch.equal(ep[:, k], st[q]), q
    o = O.evaluate(s, ens.X[:100].cpu().numpy())
    sc = 0.5 * (np.sum(np.abs(o["lap"]), axis=1) + np.sum(o["grad"] ** 2, axis=(1, 2))) + 1.0
    err = np.abs(ep[:100, 3].cpu().numpy() - o["e_loc"]) / (np.abs(o["e_loc"]) + sc)
    assert np.max(err) < (1e-9 if prec == "fp64" else 2e-3)
    # the same walkers in an ensemble that shares lanes
    small = _ensemble(ctx, s, 100, prec)
    small.run(6, 0.4, measure_every=2)
    same = torch.all((small.X == ens.X[:100]).view(100, -1), dim=1)
    # FP64 adds the pair terms in another order: parts only at a decision
    # within rounding
    assert bool(same.all()) if prec == "mixed" else int((~same).sum()) <= 1
    assert ctx.flags() == 0


@pytest.mark.parametrize("name,prec,W,spec", [("H2O", "fp64", 37889, 0), ("H2O", "mixed", 37889, 0),
                                              ("H2O+j3", "mixed", 2369, 1)])
def test_equilibration_with_one_thread_per_walker(name, prec, W, spec):
    """Device-side adaptation after k_moves: the recorded ratios are whole
    multiples of 1 / (W n_e), the widths follow the rule and the walkers are
    those of run() with these widths, refreshes included."""
    s = _system(name)
    ctx = GTOContext(s)
    if spec:
        ctx.specialize()
    ens = _ensemble(ctx, s, W, prec)
    ens.refresh_every = 3
    step, acc, widths = ens.equilibrate(7, 0.5, target=0.4, rate=0.05)
    acc, widths = acc.cpu().numpy(), widths.cpu().numpy()
    n = acc * W * s.n_e
    assert np.max(np.abs(n - np.round(n))) < 1e-6 and np.all((n > 0) & (n <= W * s.n_e))
    w = np.concatenate([[0.5], widths])
    np.testing.assert_allclose(w[1:], w[:-1] * np.exp(0.05 * (acc - 0.4)), rtol=1e-13)
    assert step == widths[-1]
    ens2 = _ensemble(ctx, s, W, prec)
    ens2.refresh_every = 3
    for k in range(7):
        ens2.run(1, float(w[k]))
    assert torch.equal(ens.X, ens2.X)
    assert torch.equal(ens.logdet(), ens2.logdet())


def test_tensor_core_energies_after_one_thread_moves():
    """The tensor-core local energy reads the state that k_moves leaves: the
    walkers are those of the CUDA-core path and the energies the oracle's."""
    s = _system("H2O")
    W, out = 37889, []
    for tc in (False, True):
        ctx = GTOContext(s)
        ctx.use_tensor_cores(tc)
        ens = _ensemble(ctx, s, W, "mixed")
        ep = torch.zeros(W, 4, dtype=torch.float64, device="cuda")
        ens.run(4, 0.4, eparts_last=ep)
        out.append((ens.X, ep, ens.logdet().clone()))
        assert ctx.flags() == 0
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][2], out[1][2])
    o = O.evaluate(s, out[1][0][:200].cpu().numpy())
    err = np.abs(out[1][1][:200, 3].cpu().numpy() - o["e_loc"])
    assert np.median(err) < 1e-4 and np.quantile(err, 0.99) < 2e-2
