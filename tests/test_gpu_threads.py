"""Calls from several host threads (ctypes drops the interpreter lock) on one
molecule, whose launches of one kernel take different amounts of shared
memory: no launch fails and each thread gets the results it gets alone."""
import threading

import pytest
import torch

from helpers import seeded_walkers
from omegaqmc_b200 import molecules as M
from omegaqmc_b200.context import GTOContext
from omegaqmc_b200.sampler import WalkerEnsemble
from omegaqmc_b200.system import build_system

pytestmark = pytest.mark.gpu


def test_launches_of_different_shared_memory():
    """FP64 H2O in CTAs of 128 and of 64 walkers, 99 and 58 KB.  A measured
    sweep is a launch of its own here, so one call makes thousands of launches
    in a row and those of the two threads interleave."""
    s = build_system(M.make_mf("H2O"), M.benchmark_params_corr(M.named_system("H2O")))
    n = 10000

    def ensembles():
        return [WalkerEnsemble(GTOContext(s), seeded_walkers(s, 33, 0.9, 3), "fp64", seed=4,
                               refresh_every=10**9, walkers_per_block=wpb) for wpb in (128, 64)]

    alone = ensembles()
    for e in alone:
        e.run(n, 0.3)
    ens, errors, gate = ensembles(), [], threading.Barrier(2)
    torch.cuda.synchronize()

    def work(e):
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                gate.wait()
                e.run(n, 0.3, stream=st)
        except Exception as ex:                     # noqa: BLE001
            errors.append(repr(ex))

    th = [threading.Thread(target=work, args=(e,)) for e in ens]
    for t in th:
        t.start()
    for t in th:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for a, b in zip(alone, ens):
        assert torch.equal(a.X, b.X) and b.ctx.flags() == 0
    # the CTA size does not enter a walker's chain
    assert torch.equal(ens[0].X, ens[1].X)
