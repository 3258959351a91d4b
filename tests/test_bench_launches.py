"""The benchmark's launch count of fused sweeps."""
import bench


class _Ens:
    def __init__(self, since):
        self.since_refresh, self.refresh_every = since, 50


def test_fused_launch_count_follows_the_chunking():
    # two 50-sweep calls, each followed by a refresh (conversion + kernel)
    assert bench.fused_launches(_Ens(0), 100) == 2 * (1 + 2)
    # 30 sweeps left in the phase: one call, refresh, then 20 more
    assert bench.fused_launches(_Ens(20), 50) == (1 + 2) + 1
    # tensor-core local energy: a sweep and an energy kernel per measurement,
    # one more sweep kernel for the two sweeps after the last measurement
    assert bench.fused_launches(_Ens(0), 50, 4, True) == 24 + (0 + 1) + 2
