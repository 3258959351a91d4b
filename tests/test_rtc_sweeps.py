"""The kernels that oqmc_specialize builds compile for sm_100a (NVRTC on the
host, no GPU): the fused sweeps and the local energy with every optional
Jastrow term and shell, and the moves alone that three-body systems add."""
import warnings

import numpy as np
import pytest

import rtc_check as R
from helpers import golden_system
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.system import build_system


def _system(name):
    if name.startswith("golden:"):
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            return golden_system(name[7:])[0]
    mol = M.named_system(name.split("+")[0])
    pc, cfg = M.benchmark_params_corr(mol), None
    if "+j3" in name:
        pc["J3_eeI"] = {p + e: 0.003 * np.arange(8.0) for e in sorted(set(mol.elements))
                        for p in ("like+", "unlike+")}
        cfg = {"J3": {"N_eI": 2, "N_ee": 2, "r_cut": 4.0}}
    return build_system(M.make_mf(name.split("+")[0]), pc, None, cfg)


def _names(n, kernels):
    return [f"{k}<{n}, {t}, {t}, {extra}OqSpecBasis>" for k, extra in kernels
            for t in ("double", "float")]


@pytest.mark.parametrize("name", ["H2", "LiH+j3", "golden:fg_shells", "golden:h2o_bspline"])
def test_specialised_kernels_compile(name):
    try:
        R._nvrtc()
    except OSError:
        pytest.skip("NVRTC not installed")
    s = _system(name)
    src = R.spec_source(s)
    ok, log, cubin = R.compile_source(src, _names(s.nocc, [("k_sweeps", ""), ("k_eloc", "")]))
    assert ok, log
    assert len(cubin) > 10000
    if "+j3" in name:
        # built without the absent terms' defines
        src = "\n".join(x for x in src.split("\n") if not x.startswith("#define OQ_GEN_"))
        ok, log, _ = R.compile_source(src, _names(s.nocc, [("k_moves", "0, "), ("k_moves", "1, ")]))
        assert ok, log
