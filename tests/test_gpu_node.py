"""Walkers next to a node of the determinant, which ``evaluate`` forms again
orbital by orbital: gradient, Laplacian and kinetic energy against an
extended-precision (x86 long double) evaluation, with several such walkers in
one tile and in a partial last tile, with and without the B-spline, three-body
and cusp terms of the general instantiation."""
import warnings

import numpy as np
import pytest

from helpers import seeded_walkers
from oracle import gto_oracle as O
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.context import GTOContext
from omegaqmc_b200.system import build_system

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
LD = np.longdouble


def _system(name):
    mol = M.named_system(name.split("+")[0])
    cusp = M.synthetic_cusp_params(mol) if "+cusp" in name else None
    pc, cfg = M.default_params_corr(mol, cusp=cusp is not None), None
    els = sorted(set(mol.elements))
    if "+bs" in name:
        pc["J2_bspline"] = {"like": np.array([0.2, 0.1, 0.05]), "unlike": np.linspace(0.4, 0.0, 9)}
        pc["J1_bspline"] = {e: np.array([-0.1, 0.05, 0.02, 0.01]) for e in els}
        cfg = {"J2": {"r_cut": 3.5}, "J1": {e: {"r_cut": 3.0} for e in els}}
    if "+j3" in name:
        rng = np.random.default_rng(4)
        pc["J3_eeI"] = {p + e: rng.normal(size=8) * 0.003 for e in els for p in ("like+", "unlike+")
                        if p + e != "like+H"}
        cfg = {"J3": {"N_eI": 2, "N_ee": 2, "r_cut": 4.0}}
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return build_system(M.make_mf(name.split("+")[0]), pc, cusp, cfg)


def _orbitals(s, x):
    """Values, gradients and Laplacians of the occupied orbitals at x (..., 3)
    in long double."""
    val, grad, lap = [], [], []
    for sh in s.shells:
        d = x - s.nuc[sh.iat].astype(LD)
        r2 = np.sum(d * d, axis=-1)
        a = sh.alpha.astype(LD)
        e = np.exp(-a * r2[..., None]) * sh.norm.astype(LD)
        R, Rp = np.sum(e, axis=-1), np.sum(-2 * a * e, axis=-1)
        Rl = np.sum((4 * a * a * r2[..., None] - 6 * a) * e, axis=-1)
        if sh.am == 0 and sh.is_cusp:
            R, Rp, Rl = O.cusp_s_vgl(np.sqrt(r2), s.cusp_rc[sh.iat], s.Z[sh.iat], R, Rp, Rl,
                                     s.cusp_q0[sh.iat], s.cusp_coeff[sh.iat].astype(LD))
        for comp in O.HARMONICS[sh.am]:
            Y, G = np.zeros_like(R), np.zeros_like(d)
            for c, *p in comp:
                Y = Y + c * np.prod([d[..., k] ** p[k] for k in range(3)], axis=0)
                for k in range(3):
                    if p[k]:
                        q = [p[j] - (j == k) for j in range(3)]
                        G[..., k] += c * p[k] * np.prod([d[..., j] ** q[j] for j in range(3)], axis=0)
            val.append(R * Y)
            grad.append((Rp * Y)[..., None] * d + R[..., None] * G)
            lap.append((Rl + 2 * sh.am * Rp) * Y)
    C = np.asarray(s.C).astype(LD)
    f = lambda q: np.sum(q[..., None] * C, axis=-2)                     # noqa: E731
    return (f(np.stack(val, -1)), np.stack([f(np.stack([g[..., k] for g in grad], -1))
                                            for k in range(3)], -1), f(np.stack(lap, -1)))


def _inverse(S):
    n = len(S)
    A = np.concatenate([S, np.eye(n, dtype=LD)], axis=1)
    for k in range(n):
        p = k + int(np.argmax(np.abs(A[k:, k])))
        A[[k, p]] = A[[p, k]]
        A[k] /= A[k, k]
        for i in range(n):
            if i != k:
                A[i] -= A[i, k] * A[k]
    return A[:, n:]


def exact(s, X):
    """(grad, lap, e_ke, sum of squared gradients) of log|psi| in long double;
    the Jastrow part, smooth across the node, from the FP64 oracle."""
    v, g, l = _orbitals(s, X.astype(LD))
    gs, lp = np.zeros(X.shape, dtype=LD), np.zeros(X.shape[:2], dtype=LD)
    for w in range(len(X)):
        for sp in (0, 1):
            A = _inverse(v[w, sp::2])
            gs[w, sp::2] = np.einsum("mi,imc->ic", A, g[w, sp::2])
            lp[w, sp::2] = np.einsum("mi,im->i", A, l[w, sp::2])
    gj, lj = (q.astype(LD) for q in O.jastrow_vgl(s, X))
    ke = -0.5 * (np.sum(lp + lj, axis=1) + np.sum(2 * gs * gj + gj * gj, axis=(1, 2)))
    return gs + gj, lp - np.sum(gs * gs, -1) + lj, ke, np.sum((gs + gj) ** 2, axis=(1, 2))


def near_nodes(s, n, seed):
    """n walkers next to a node of the up determinant: on the line between two
    walkers of opposite sign, and with two up electrons 1e-6 apart."""
    rng = np.random.default_rng(seed)
    X = seeded_walkers(s, 40 * n, 0.9, seed)

    def det(x):
        return np.linalg.slogdet(np.asarray(O.mo_value(s, x[None])[0, 0::2]))[0]

    out = []
    for k in range(0, len(X) - 1, 2):
        if len(out) == n:
            break
        if len(out) % 3 == 2:
            x = X[k].copy()
            u = rng.standard_normal(3)
            x[2] = x[0] + 1e-6 * u / np.linalg.norm(u)
            out.append(x)
            continue
        a, b = X[k], X[k + 1]
        sa = det(a)
        if det(b) == sa:
            continue
        lo, hi = 0.0, 1.0
        for _ in range(60):
            t = 0.5 * (lo + hi)
            lo, hi = (t, hi) if det(a + t * (b - a)) == sa else (lo, t)
        out.append(a + (lo + 10.0 ** -rng.uniform(7.3, 8.5)) * (b - a))
    assert len(out) == n
    return np.array(out)


@pytest.mark.parametrize("name", ["H2O", "LiH", "N2", "H2O_dimer", "H2O+bs", "H2O+j3", "LiH+cusp"])
def test_walkers_next_to_a_node(name):
    s = _system(name)
    ctx = GTOContext(s)
    W, n = 133, 12
    X = seeded_walkers(s, W, 0.9, 11)
    near = near_nodes(s, n, 23)
    # several in the first tile, one alone, several in the partial last one
    at = np.r_[0, 1, 2, 5, 6, 40, 77, 78, W - 4, W - 3, W - 2, W - 1]
    X[at] = near
    r = {k: v.cpu().numpy() for k, v in ctx.evaluate(X).items()}
    grad, lap, ke, g2 = exact(s, near)
    # the branch's own condition, well inside it
    assert np.all(g2 > 4e5 * np.abs(2 * ke)), np.sort(np.float64(g2 / np.abs(2 * ke)))
    # what FP64 determines: the inverse's relative error is eps times its
    # condition, of order |gradient|, so g carries eps g^2 and ke carries
    # eps g2; 200 leaves room for N^2 terms and orbital-scale factors
    scale = np.sqrt(np.float64(g2))
    tol = 200 * EPS * scale
    for k, ref in (("grad", grad), ("lap", lap)):
        err = np.abs(r[k][at] - np.float64(ref)).reshape(n, -1).max(axis=1)
        size = np.abs(np.float64(ref)).reshape(n, -1).max(axis=1)
        assert np.all(err < (1e-9 + tol) * size), (k, err / size, tol)
    err = np.abs(r["e_ke"][at] - np.float64(ke))
    assert np.all(err < 200 * EPS * np.float64(g2)), (err, np.float64(g2))
    # outputs asked for or not, and the other walkers of their tiles
    r1 = {k: v.cpu().numpy() for k, v in ctx.evaluate(X, want_grad=False, want_lap=False).items()}
    assert np.array_equal(r1["e_ke"], r["e_ke"]) and np.array_equal(r1["e_loc"], r["e_loc"])
    rest = np.setdiff1d(np.arange(W), at)
    alone = ctx.evaluate(X[rest])
    for k in ("grad", "lap", "e_ke", "logpsi"):
        assert np.array_equal(r[k][rest], alone[k].cpu().numpy()), k
    o = O.evaluate(s, X[rest])
    fine = np.sqrt(np.sum(o["grad"] ** 2, axis=(1, 2))) < 1e3
    e = np.abs(r["grad"][rest] - o["grad"]) / (np.abs(o["grad"]) + 1)
    assert np.max(e[fine]) < 1e-10
