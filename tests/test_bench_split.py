"""The benchmark's launch count on the split path, by route."""
from types import SimpleNamespace as N

import bench


def _ens(W, precision, nocc):
    return N(W=W, precision=precision, since_refresh=0, refresh_every=50, ctx=N(nocc=nocc))


def test_split_launches_follow_the_route():
    fused = 2 * (1 + 2)                       # two 50-sweep calls, each with a refresh
    assert bench.split_launches(_ens(65536, "mixed", 5), 100, False, False) == fused
    assert bench.split_launches(_ens(65536, "fp64", 5), 100, False, False) == fused
    # table-driven, one thread per walker: two conversions, moves and energies
    assert bench.split_launches(_ens(65536, "mixed", 5), 100, True, False) == 2 * (2 + 100 + 2)
    assert bench.split_launches(_ens(37888, "mixed", 5), 100, True, False) == fused
    assert bench.split_launches(_ens(65536, "mixed", 2), 100, True, False) == fused
    # FP64, eight and more orbitals: energies apart
    assert bench.split_launches(_ens(65536, "fp64", 10), 100, False, False) == 2 * (100 + 2)
    assert bench.split_launches(_ens(65536, "mixed", 10), 100, False, False) == fused
    assert bench.split_launches(_ens(2048, "mixed", 5), 100, False, True) == 2 * (100 + 2)
