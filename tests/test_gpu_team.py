"""The tile kernels of the FP64 evaluation (one thread per walker and
electron) at the sizes where a tile can go wrong: one walker, a partial tile,
a tile's edge, more tiles than SMs, every determinant size the padding and
the CTA size depend on, and basis entries of three and four contraction
columns (split in the packed tables).  Oracle tolerances as in
test_gpu_eval.py: 1e-10 of |value| + 1, kinetic energies of the magnitude of
the terms they sum."""
import numpy as np
import pytest

from helpers import seeded_walkers
from oracle import gto_oracle as O
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.context import GTOContext
from omegaqmc_b200.sampler import WalkerEnsemble
from omegaqmc_b200.system import MeanField, Mole, build_shells, build_system

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _cluster(n_el, basis):
    """Closed-shell cluster of Be / He / C atoms with n_el electrons and seeded orbitals."""
    z = {"Be": 4, "He": 2, "C": 6}
    syms, left = [], n_el
    while left:
        s = "C" if left >= 6 else "Be" if left >= 4 else "He"
        syms.append(s)
        left -= z[s]
    atoms = [(s, (1.9 * (i % 3), 2.1 * (i // 3), 0.4 * (-1) ** i)) for i, s in enumerate(syms)]
    return Mole(atoms, {s: basis(s) for s in set(syms)}, unit="Bohr")


def _system(nocc, basis=M.ccpvdz_shaped):
    mol = _cluster(2 * nocc, basis)
    rng = np.random.default_rng(nocc)
    sh = build_shells(mol)
    nbf = sh[-1].isgs + sh[-1].nsgs
    C = np.linalg.qr(rng.standard_normal((nbf, nbf)))[0][:, :nocc]
    return build_system(MeanField(mol, C), M.default_params_corr(mol))


def _columns(sym):
    """A basis with general contractions of three and four columns."""
    a = [30.0, 6.0, 1.5, 0.4]
    return [[0] + [[x, 0.1 * k + 0.1, 0.5 - 0.1 * k, (-1.0) ** k * 0.3] for k, x in enumerate(a)],
            [1] + [[x, 0.2, 0.1 * k, 0.4 - 0.1 * k, (-1.0) ** k] for k, x in enumerate(a[1:])],
            [2, [0.8, 1.0]]]


def _err(a, b):
    return float(np.max(np.abs(a.cpu().numpy() - b) / (np.abs(b) + 1.0)))


def _check(s, W):
    ctx = GTOContext(s)
    X = seeded_walkers(s, W, 0.9, 100 + W)
    r, o = ctx.evaluate(X), O.evaluate(s, X)
    # determinants of seeded orbitals can be near-singular: relative errors
    # grow with the condition number, so compare where it is moderate
    g2 = np.sqrt(np.sum(o["grad"] ** 2, axis=(1, 2)))
    fine = g2 < 1e3
    assert fine.mean() > 0.9 or W < 20
    for k in ("e_ee", "e_en"):
        assert _err(r[k], o[k]) < TOL, k
    for k in ("logpsi", "grad", "lap"):
        assert _err(r[k][fine], o[k][fine]) < TOL, (k, _err(r[k][fine], o[k][fine]))
    sc = 0.5 * (np.sum(np.abs(o["lap"]), axis=1) + g2 ** 2) + 1.0
    for k in ("e_ke", "e_loc"):
        e = np.abs(r[k].cpu().numpy() - o[k]) / (np.abs(o[k]) + sc)
        assert np.max(e[fine]) < TOL, k
    assert _err(ctx.log_psi(X)[fine], o["logpsi"][fine]) < TOL
    mo = ctx.mo_values(X)
    assert mo.shape == (W, s.n_e, s.nocc)
    # the refreshed sampler state holds the same log|det| and inverses
    ens = WalkerEnsemble(ctx, X, "fp64", seed=1)
    st = ens.state_evaluate()
    assert _err(st["grad"][fine], o["grad"][fine]) < TOL
    assert _err(st["logpsi"][fine], o["logpsi"][fine]) < TOL
    assert ctx.flags() == 0


@pytest.mark.parametrize("name,W", [("H2", 1), ("H2", 63), ("H2", 65), ("H2", 40000),
                                    ("LiH", 3), ("H2O", 1), ("H2O", 33), ("H2O", 20001),
                                    ("N2", 5), ("H2O_dimer", 17)])
def test_tiles_match_oracle(name, W):
    mf = M.make_mf(name)
    _check(build_system(mf, M.default_params_corr(mf.mol)), W)


@pytest.mark.parametrize("nocc", [3, 4, 6, 8, 12, 14, 16])
def test_determinant_sizes_match_oracle(nocc):
    _check(_system(nocc), 37)


def test_wide_contractions_match_oracle():
    _check(_system(3, _columns), 50)


@pytest.mark.parametrize("name,extra,W", [("H2", None, 1), ("H2O", "bspline", 5),
                                          ("H2O_dimer", "bspline", 3), ("LiH", "j3", 2),
                                          ("H2O", "j33", 7)])
def test_parameter_derivatives_raw_and_mapped(name, extra, W):
    """One warp per walker, four to a CTA: the raw derivatives against the
    oracle (a wide and a narrow determinant, both spline blocks, three-body
    orders 2 and 3 with more gammas than lanes), and the mapped form against
    raw_to_flat of the raw one."""
    import ctypes
    import torch
    from omegaqmc_b200.context import _dptr, _stream_ptr
    from omegaqmc_b200.optim import raw_to_flat, walker_derivatives
    mol = M.named_system(name)
    pc, cfg = M.default_params_corr(mol), None
    els = sorted(set(mol.elements))
    if extra == "bspline":
        pc["J2_bspline"] = {"like": np.array([0.2, 0.1, 0.05]), "unlike": np.linspace(0.4, 0.0, 9)}
        pc["J1_bspline"] = {e: np.array([-0.1, 0.05, 0.02, 0.01]) for e in els}
        cfg = {"J2": {"r_cut": 3.5}, "J1": {e: {"r_cut": 3.0} for e in els}}
    elif extra:
        k = 2 if extra == "j3" else 3
        rng = np.random.default_rng(6)
        pc["J3_eeI"] = {p + e: rng.normal(size={2: 8, 3: 26}[k]) * 0.01 for e in els
                        for p in ("like+", "unlike+") if p + e != "like+" + els[0]}
        cfg = {"J3": {"N_eI": k, "N_ee": k, "r_cut": 4.5}}
    import warnings
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        s = build_system(M.make_mf(name), pc, None, cfg)
    ctx = GTOContext(s)
    X = ctx.walkers_tensor(seeded_walkers(s, W, 0.9, 7))
    grad = ctx.evaluate(X)["grad"]
    n = ctx.lib.oqmc_param_count(ctx._h)
    dl = torch.full((W, n), np.nan, dtype=torch.float64, device="cuda")
    de = dl.clone()
    ctx._check(ctx.lib.oqmc_param_derivs(ctx._h, _dptr(X), W, _dptr(grad), _dptr(dl), _dptr(de),
                                         _stream_ptr(None)))
    rl, re_ = O.param_derivatives(s, X.cpu().numpy())
    assert np.max(np.abs(dl.cpu().numpy() - rl) / (np.abs(rl).max(axis=0) + 1.0)) < 1e-10
    assert np.max(np.abs(de.cpu().numpy() - re_) / (np.abs(re_).max(axis=0) + 1.0)) < 1e-9
    e, fl, fe = walker_derivatives(ctx, X, pc)
    ml, me = raw_to_flat(dl.cpu().numpy(), pc, s), raw_to_flat(de.cpu().numpy(), pc, s)
    # the same products summed in another order
    assert np.max(np.abs(fl - ml) / (np.abs(ml).max(axis=0) + 1.0)) < 1e-13
    assert np.max(np.abs(fe - me) / (np.abs(me).max(axis=0) + 1.0)) < 1e-13
    assert e.shape == (W,) and fl.shape == fe.shape == ml.shape
    assert ctx.lib.oqmc_param_derivs_mapped(ctx._h, _dptr(X), W, _dptr(grad), None, None, 0, None,
                                            None, None, ctypes.c_void_p(0)) == -1


@pytest.mark.parametrize("name,prec,sizes", [("H2", "fp64", (1, 70, 40000)),
                                             ("LiH", "fp64", (2, 33, 5000)),
                                             ("H2O", "fp64", (3, 65, 20001)),
                                             ("H2O", "mixed", (3, 500)),
                                             ("H2O_dimer", "fp64", (1, 17))])
def test_all_electron_steps_do_not_depend_on_the_tile(name, prec, sizes):
    """A walker's chain depends on its index and the seed, not on the tile it
    shares: the first walkers of ensembles whose tiles differ (one warp up to
    full CTAs, partial last tiles) agree, and the last local energies and
    log|det| match the oracle at the final walkers."""
    import torch
    mf = M.make_mf(name)
    s = build_system(mf, M.default_params_corr(mf.mol))
    X = seeded_walkers(s, max(sizes), 0.8, 5)
    runs = []
    for W in sizes:
        ctx = GTOContext(s)
        ctx.set_move_kind(1)
        ens = WalkerEnsemble(ctx, X[:W], prec, seed=4, refresh_every=10**9)
        ep = torch.zeros(W, 4, dtype=torch.float64, device="cuda")
        sums = ens.run(6, 0.12, measure_every=2, eparts_last=ep)
        assert torch.all(sums[:, 6] == W) and torch.all(sums[:, 5] % s.n_e == 0)
        assert abs(float(sums[-1, 3]) - float(ep[:, 3].sum())) < 1e-9 * float(ep[:, 3].abs().sum())
        m = min(W, 100)
        o = O.evaluate(s, ens.X[:m].cpu().numpy())
        sc = 0.5 * (np.sum(np.abs(o["lap"]), axis=1) + np.sum(o["grad"] ** 2, axis=(1, 2))) + 1.0
        err = np.abs(ep[:m, 3].cpu().numpy() - o["e_loc"]) / (np.abs(o["e_loc"]) + sc)
        assert np.max(err) < (1e-10 if prec == "fp64" else 2e-3)
        ld = ens.logdet()[:m].cpu().numpy()
        assert np.max(np.abs(ld - O.log_slater(s, ens.X[:m].cpu().numpy())) / (np.abs(ld) + 1)) < TOL
        ens.run(1, 0.12)                       # a step after the last measurement
        assert ctx.flags() == 0
        runs.append(ens.X)
    for a, b in zip(runs, runs[1:]):
        assert torch.equal(a, b[: a.shape[0]])
    assert not torch.equal(runs[-1], torch.as_tensor(X, device="cuda"))


@pytest.mark.parametrize("W", [1, 33, 4097])
def test_f_and_g_shell_values_match_oracle(W):
    """The value path of f and g shells (mo_values, log_psi, the refresh)
    forms no harmonic gradients; its values are evaluate's."""
    from helpers import golden_system
    s, _ = golden_system("fg_shells")
    ctx = GTOContext(s)
    X = seeded_walkers(s, W, 0.9, 17)
    m = min(W, 200)
    mo = ctx.mo_values(X)[:m].cpu().numpy()
    ref = O.mo_value(s, X[:m])
    assert np.max(np.abs(mo - ref) / (np.abs(ref) + 1.0)) < TOL
    lp, ev = ctx.log_psi(X).cpu().numpy(), ctx.evaluate(X)["logpsi"].cpu().numpy()
    assert np.max(np.abs(lp - ev) / (np.abs(ev) + 1.0)) < 1e-12
    ens = WalkerEnsemble(ctx, X, "fp64", seed=1)
    ld = ens.logdet()[:m].cpu().numpy()
    assert np.max(np.abs(ld - O.log_slater(s, X[:m])) / (np.abs(ld) + 1.0)) < TOL


@pytest.mark.parametrize("name,bs,W", [("H2", False, 4001), ("H2", False, 4000), ("LiH", False, 5601),
                                       ("H2O", True, 10501), ("H2", True, 4097)])
def test_raw_derivatives_of_many_walkers(name, bs, W):
    """One thread per walker above 4,000 walkers and 400 per pair term (140
    with B-splines; H2 has 5 terms, LiH 14, H2O 75): against the oracle on both
    sides of the line, and the last walkers of a partial CTA."""
    import torch
    from omegaqmc_b200.context import _dptr, _stream_ptr
    mol = M.named_system(name)
    pc, cfg = M.default_params_corr(mol), None
    els = sorted(set(mol.elements))
    if bs:
        pc["J2_bspline"] = {"like": np.array([0.2, 0.1, 0.05]), "unlike": np.linspace(0.4, 0.0, 9)}
        pc["J1_bspline"] = {e: np.array([-0.1, 0.05, 0.02, 0.01]) for e in els}
        cfg = {"J2": {"r_cut": 3.5}, "J1": {e: {"r_cut": 3.0} for e in els}}
    import warnings
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        s = build_system(M.make_mf(name), pc, None, cfg)
    ctx = GTOContext(s)
    X = ctx.walkers_tensor(seeded_walkers(s, W, 0.9, 7))
    grad = ctx.evaluate(X)["grad"]
    n = ctx.lib.oqmc_param_count(ctx._h)
    dl = torch.full((W + 1, n), np.nan, dtype=torch.float64, device="cuda")
    de = dl.clone()
    ctx._check(ctx.lib.oqmc_param_derivs(ctx._h, _dptr(X), W, _dptr(grad), _dptr(dl), _dptr(de),
                                         _stream_ptr(None)))
    assert bool(torch.isnan(dl[W]).all()) and bool(torch.isnan(de[W]).all())
    pick = np.r_[0:40, W - 40:W]
    rl, re_ = O.param_derivatives(s, X.cpu().numpy()[pick])
    assert np.max(np.abs(dl.cpu().numpy()[pick] - rl) / (np.abs(rl).max(axis=0) + 1.0)) < 1e-10
    assert np.max(np.abs(de.cpu().numpy()[pick] - re_) / (np.abs(re_).max(axis=0) + 1.0)) < 1e-9
    # the mapped form keeps a warp per walker: the same numbers, other sums
    from omegaqmc_b200.optim import raw_to_flat, walker_derivatives
    e, fl, fe = walker_derivatives(ctx, X, pc)
    ml = raw_to_flat(dl[:W].cpu().numpy(), pc, s)
    me = raw_to_flat(de[:W].cpu().numpy(), pc, s)
    assert np.max(np.abs(fl - ml) / (np.abs(ml).max(axis=0) + 1.0)) < 1e-12
    assert np.max(np.abs(fe - me) / (np.abs(me).max(axis=0) + 1.0)) < 1e-12
