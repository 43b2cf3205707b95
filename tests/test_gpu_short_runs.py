"""Short queued runs with a FarFieldCBS sensor: every photon's history tracked, or the photons
the grid reads replayed, by how many those are and how long the paths get."""
import pytest

import luminis_mc_b200 as lm
from luminis_mc_b200 import workloads as W
from tests.test_gpu_variants import assert_same_run, run_tallies

pytestmark = pytest.mark.gpu


def _long(n):
    return dict(W.mie_long_paths(n, 41), max_events=4000)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("make,n,replays", [
    (W.mie_cbs_small, 1, 1), (W.mie_cbs_small, 300, 1), (W.mie_cbs_small, 3000, 0), (W.mie_cbs_small, 18_944, 0),
    (W.mie_cbs_small, 18_945, 1), (_long, 300, 1), (_long, 12_000, 1), (W.bilayer_hg, 300, 1), (W.bilayer_hg, 9001, 0)])
def test_short_runs_replay_where_little_is_read(make, n, replays, precision, cuda):
    """A grid of 0.1 rad reads 1 % of the photons, of 0.02 rad 0.04 %: tracking every event of
    the longest path pays for many of them only.  Same tallies either way."""
    spec = make(n, 41) if make is not _long else make(n)
    got, want = run_tallies(spec, precision), run_tallies(spec, precision, no_replay=True)
    assert got[0]["replay_launches"] == replays and want[0]["replay_launches"] == 0
    assert_same_run(got, want, 1e-12)


@pytest.mark.parametrize("n,replays", [(300, 1), (6000, 0)])
def test_short_sweeps_and_derivatives(n, replays, cuda):
    from luminis_mc_b200.adjoint import AdjointTransport
    from luminis_mc_b200.sweep import SweepRun
    import numpy as np
    cfg, _, keep = W.build(lm, W.bilayer_hg(n, 43))
    tr = AdjointTransport(cfg, radial_sensor=1, radial_bins=20, radial_max=5.0)
    stats = [x for x in tr.run(n, 43) if isinstance(x, dict)][0]
    tr.close()
    assert stats["replay_launches"] == replays
    sweep = SweepRun(W.build_mie_sweep(lm, [W.mie_sweep(i, seed=3, count=3) for i in range(3)]), device="cuda:0")
    sweep.set_photons(np.full(3, n // 3, np.uint64))
    assert sweep.run(43)["replay_launches"] == replays
    assert sweep.run_adjoint(43)[1]["replay_launches"] == replays
