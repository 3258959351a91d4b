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
