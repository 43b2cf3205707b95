"""Scenes with sensor planes inside the sample: hits buffered per warp, and the photons a
FarFieldCBS grid reads run again, against every hit processed on the spot (`no_replay`)."""
import pytest

from luminis_mc_b200 import workloads as W
from tests.test_gpu_variants import TOL, assert_same_run, run_tallies

pytestmark = pytest.mark.gpu


def _planes(n, planes, cone=False, first=None, absorption=False):
    """Fluence at `planes` depths within one mean free path, beside the surface cone."""
    spec = W.bilayer_rgd_mie(n, 31)
    spec["sensors"] = spec["sensors"][:1] if cone else []
    if first is not None:
        spec["sensors"].insert(0, first)
    for i in range(planes):
        spec["sensors"].append({"kind": "planar_fluence", "z": 0.006 * (i + 1), "len_x": 4.0, "len_y": 4.0,
                                "len_t": 0.0, "dx": 0.25, "dy": 0.25, "d_t": 0.0, "absorb": False})
    if absorption:
        spec["absorption"] = {"radius": 3.0, "depth": 2.0, "d_r": 0.25, "d_z": 0.1}
    return spec


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,planes,block", [(33, 8, 32), (40_001, 8, 0), (40_001, 2, 96)])
def test_buffers_filled_many_times_over_lose_no_hit(n, planes, block, precision, cuda):
    """Planes closer than a flight: an event adds up to eight hits a lane, so that a warp's
    fill passes 32 in most events and by any amount.  Every lane of the warp has to read the
    same fill; the counts of three runs equal the on-the-spot ones."""
    spec = _planes(n, planes)
    want = run_tallies(spec, precision, no_replay=True)
    assert sum(want[0]["hits"]) > n
    for _ in range(3):
        assert_same_run(run_tallies(spec, precision, block_size=block), want, TOL[precision])
