"""The allocation-free entry point judges the kernels that the call launches:
with the device's stack limit lowered (this process's own context) below what
the general instantiations and the separate local-energy kernel need, calls
whose own kernels fit still run, from the first call on."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

# Run in a fresh process, before anything has raised the limit.
_FRESH = r"""
import ctypes, json, sys
import torch
sys.path[:0] = [sys.argv[1], sys.argv[2]]
from helpers import seeded_walkers
from omegaqmc_b200 import _lib as L
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.context import GTOContext
from omegaqmc_b200.system import build_system

lib = L.load()
torch.zeros(1, device="cuda")
rt = ctypes.CDLL("libcudart.so.12")
lim = ctypes.c_size_t()
rt.cudaDeviceSetLimit(0, ctypes.c_size_t(160))
rt.cudaDeviceGetLimit(ctypes.byref(lim), 0)
out = {"limit": lim.value}
s = build_system(M.make_mf("H2O"), M.benchmark_params_corr(M.named_system("H2O")))
p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)
st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def call(move, spec, prec, W=64):
    ctx = GTOContext(s)
    ctx.set_move_kind(move)
    if spec:
        ctx.specialize()
    X = torch.tensor(seeded_walkers(s, W, 0.9, 2), dtype=torch.float64, device="cuda")
    X0 = X.clone()
    sums = torch.zeros(3, 8, dtype=torch.float64, device="cuda")
    rc = lib.oqmc_sweeps_noalloc(ctx._h, p(X), W, prec, 3, 1, 0.2, ctypes.c_uint64(1),
                                 ctypes.c_uint64(0), p(sums), None, None, st)
    torch.cuda.synchronize()
    rt.cudaDeviceGetLimit(ctypes.byref(lim), 0)
    return [rc, lib.oqmc_last_error(ctx._h).decode(), bool(torch.equal(X, X0)), lim.value]


out["alle_fp64"] = call(1, 0, L.PREC_FP64)
out["sweeps_spec_mixed"] = call(0, 1, L.PREC_MIXED)
out["sweeps_spec_fp64"] = call(0, 1, L.PREC_FP64)
# the table-driven FP64 sweeps need more than that and are refused
out["sweeps_fp64"] = call(0, 0, L.PREC_FP64)
print("RESULT " + json.dumps(out))
"""


def test_the_launched_kernels_are_judged():
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", _FRESH, here, os.path.dirname(here)],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    line = [x for x in r.stdout.splitlines() if x.startswith("RESULT ")][-1]
    out = json.loads(line[len("RESULT "):])
    if out["limit"] > 200:
        pytest.skip(f"the stack limit cannot be lowered below {out['limit']} B here")
    for k in ("alle_fp64", "sweeps_spec_mixed", "sweeps_spec_fp64"):
        rc, err, same, lim = out[k]
        assert rc == 0 and not same and lim == out["limit"], (k, out[k])
    rc, err, same, lim = out["sweeps_fp64"]
    assert rc == -6 and "local memory" in err and same, out["sweeps_fp64"]
