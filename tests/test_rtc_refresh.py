"""The generated kernels' FP64 refresh of the inverses evaluates every orbital
coefficient; the moves leave out those at round-off."""
import os
import re

import numpy as np
import pytest

import rtc_check as R
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.system import MeanField, build_system


def _terms(src, name):
    """The coefficients of the generated function ``name``, per orbital."""
    body = re.split(r"__device__|\n};", src.split(f"void {name}(")[1])[0]
    return [(int(m), float(c)) for m, c in
            re.findall(r"mv\[(\d+)\] \+= \(T\)\(([-0-9.eE+]+)\)", body)]


@pytest.mark.parametrize("name,small", [("H2O", None), ("LiH", 3e-13), ("H2", 0.0)])
def test_refresh_keeps_every_coefficient(name, small):
    mf = M.make_mf(name)
    C = np.array(mf.mo_coeff)
    nocc = mf.mol.tot_electrons() // 2
    if small is not None:
        C[-1, :nocc] = small * np.abs(C[:, :nocc]).max(axis=0)
        mf = MeanField(mf.mol, C, mf.mo_occ)
    s = build_system(mf, M.benchmark_params_corr(mf.mol))
    src = R.batch_source([s])
    want = sorted((m, float(c)) for m in range(s.nocc) for c in np.asarray(s.C)[:, m] if c != 0.0)
    assert sorted(_terms(src, "mo_val_full")) == want
    kept = _terms(src, "mo_val")
    assert len(kept) < len(want) if name == "H2O" or small else len(kept) == len(want)


def test_batch_refresh_uses_it():
    src = open(os.path.join(R.CSRC, "oqmc_batch.cuh")).read()
    refresh = src[src.index("FP64 refresh of the spin blocks: both"):src.index("oq_invert<")]
    assert "B::template mo_val_full<double, double>" in refresh
    assert "mo_val<" not in refresh
