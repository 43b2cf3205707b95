"""Scenes with sensor planes inside the sample: hits buffered per warp, and the photons a
FarFieldCBS grid reads run again, against every hit processed on the spot (`no_replay`)."""
import numpy as np
import pytest

import luminis_mc_b200 as lm
from luminis_mc_b200 import workloads as W
from luminis_mc_b200.device import DeviceRun
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


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("make,n", [(lambda n: _planes(n, 3, cone=True), 200_003), (lambda n: _planes(n, 2), 2000),
                                    (lambda n: W.mie_cbs_small(n, 31), 20_000)],
                         ids=["planes_and_cone", "planes", "queue"])
def test_a_captured_run_survives_larger_runs(make, n, precision, cuda):
    """The queue and the warps' buffers grow with the run.  A graph captured after a run of
    its size holds their address: it still gives the same run when larger runs on the handle
    have outgrown them, and so does one captured after that."""
    import torch
    spec = make(n)
    stats, want = run_tallies(spec, precision)
    cfg, _, keep = W.build(lm, spec)
    run = DeviceRun(cfg)
    stream = torch.cuda.Stream()

    def capture():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run.transport.run_device(run.tallies.data_ptr(), n, spec["seed"], want_stats=False,
                                     precision=precision, stream=stream.cuda_stream)
        return graph

    run.run(n, 1, precision=precision)
    graphs = [capture()]
    for larger in (2 * n, 5 * n):
        assert run.run(larger, 2, precision=precision)[0]["error_flags"] == 0
        graphs.append(capture())
    for graph in graphs:
        run.zero()
        graph.replay()
        for x, y in zip(run.host_tallies(), want):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-12 * max(np.abs(y).max(), 1e-300))
    del graph, graphs
    run.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("batch", [0, 60_000])
def test_the_rerun_takes_every_photon_the_cone_sees(batch, precision, cuda):
    """The cone's filter is its grid, so every photon it detects is listed, once, and run
    again; a rerun that left the listed walk would raise an error flag."""
    stats, _ = run_tallies(_planes(200_003, 2, cone=True), precision, batch_photons=batch)
    assert stats["replay_launches"] == (4 if batch else 1) and stats["error_flags"] == 0
    assert stats["replayed"] == stats["detected"] == stats["hits"][0] > 100


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_the_rerun_deposits_nothing(precision, cuda):
    """The first walk filled the Absorption grid; the photons run again for the cone must not
    fill it once more.  Grid: a cell's ~10^7 binary64 deposits in another order (1e-9 is 10^3
    times their sum's random-walk error); a second deposit of the ~1 % of photons that are
    run again is 10^6 times more."""
    spec = _planes(200_003, 2, cone=True, absorption=True)
    got, want = run_tallies(spec, precision), run_tallies(spec, precision, no_replay=True)
    assert got[0]["replay_launches"] == 1 and want[0]["replay_launches"] == 0
    assert_same_run((got[0], got[1][:-1]), (want[0], want[1][:-1]), TOL[precision])
    np.testing.assert_allclose(got[1][-1], want[1][-1], rtol=0, atol=1e-9 * want[1][-1].max())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_cone_on_a_plane_above_the_surface_stays_on_the_spot(precision, cuda):
    """Planes within 1e-9 of one another are one, at the first one's depth: a cone grouped
    onto a plane just inside the sample can see a photon more than once, so its photons
    cannot be listed and run again."""
    above = {"kind": "planar_fluence", "z": 5e-10, "len_x": 4.0, "len_y": 4.0, "len_t": 0.0, "dx": 0.25,
             "dy": 0.25, "d_t": 0.0, "absorb": False}
    spec = _planes(200_003, 2, cone=True, first=above)
    got, want = run_tallies(spec, precision), run_tallies(spec, precision, no_replay=True)
    assert got[0]["replay_launches"] == 0 and got[0]["hits"][1] > 0
    assert_same_run(got, want, 1e-12)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("make,n", [(lambda n: _planes(n, 3, cone=True), 200_003), (lambda n: _planes(n, 3), 30_001),
                                    (lambda n: W.bilayer_rgd_mie(n, 31), 60_001), (W.mie_cbs_small, 9001)],
                         ids=["planes_and_cone", "planes", "queue", "short_run"])
def test_tallies_do_not_depend_on_the_route(make, n, precision, cuda):
    """The routes' kernels round a hit's binary32 arithmetic alike: their tallies differ by
    the order of the binary64 sums alone (1e-12 of the largest bin; another binary32 rounding
    of every hit's products would be 1e-8 and more)."""
    spec = make(n)
    want = run_tallies(spec, precision)
    for options in ({"no_replay": True}, {"blocks_per_sm": 2}, {"stage_tables": True}):
        assert_same_run(run_tallies(spec, precision, **options), want, 1e-12)


def _long_paths(n, max_events, cone):
    spec = W.mie_long_paths(n, 31)
    spec["max_events"] = max_events
    plane = {"kind": "planar_fluence", "z": 0.1, "len_x": 4.0, "len_y": 4.0, "len_t": 0.0, "dx": 0.25, "dy": 0.25,
             "d_t": 0.0, "absorb": False}
    spec["sensors"] = ([spec["sensors"][0]] if cone else []) + [plane]
    return spec


@pytest.mark.parametrize("precision,n,max_events,reruns", [
    ("fp32", 200_003, 1000, 1), ("fp32", 200_003, 4000, 0), ("fp64", 110_001, 1000, 1), ("fp64", 110_001, 4000, 0)])
def test_runs_over_long_paths_stay_on_the_spot(precision, n, max_events, reruns, cuda):
    """The photons it takes for the buffers to pay grow with the longest path: the same
    photons are listed and run again with paths to 1000 events, not with paths to 4000
    (22.7 ms against 16.9 in binary32).  Same tallies either way."""
    spec = _long_paths(n, max_events, True)
    got, want = run_tallies(spec, precision), run_tallies(spec, precision, no_replay=True)
    assert got[0]["replay_launches"] == reruns
    assert_same_run(got, want, 1e-12)


@pytest.mark.parametrize("n", [37_888, 37_889, 187_206, 187_207])
def test_both_sides_of_the_rule_without_a_cone(n, cuda):
    """Binary32 without a FarFieldCBS sensor: 256 and 40 sqrt(1000) photons per SM (148)."""
    spec = _long_paths(n, 1000, False)
    assert_same_run(run_tallies(spec, "fp32"), run_tallies(spec, "fp32", no_replay=True), 1e-12)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_one_block_per_sm_of_buffers_loses_no_hit(precision, cuda):
    """The most photons that go through the buffers at one block per SM, eight planes."""
    spec = _planes(37_001, 8)
    assert_same_run(run_tallies(spec, precision), run_tallies(spec, precision, no_replay=True), TOL[precision])
