"""The digest under which run_simulation_parallel keeps its last scene: equal for scenes of
equal parameters and tables, wherever their arrays lie, and different for any other."""
import copy

import pytest

import luminis_mc_b200 as lm
from luminis_mc_b200 import workloads as W
from luminis_mc_b200.simulation import _scene_digest, scene_desc


def _digest(spec):
    cfg, _, keep = W.build(lm, spec)
    return _scene_digest(scene_desc(cfg))


@pytest.mark.parametrize("make", [W.mie_cbs_small, W.bilayer_rgd_mie, W.bilayer_hg, W.mixture_bilayer])
def test_equal_scenes_share_a_digest(make):
    assert _digest(make(1000, 1)) == _digest(make(2000, 2))       # photons and seed are the call's


@pytest.mark.parametrize("change", [
    lambda s: s["media"][0].update(mu_a=0.02), lambda s: s["media"][0].update(mfp=0.2),
    lambda s: s["phases"][0].update(radius=0.51e-3), lambda s: s["media"][0].update(radius=0.51e-3),
    lambda s: s["phases"][0].update(nDiv=999), lambda s: s["sensors"][0].update(d_theta=2e-3),
    lambda s: s["laser"].update(m=0j, n=1 + 0j), lambda s: s.update(n_host=1.0)])
def test_any_changed_parameter_or_table_changes_the_digest(change):
    spec = W.mie_cbs_small(1000, 1)
    other = copy.deepcopy(spec)
    change(other)
    assert _digest(spec) != _digest(other)
