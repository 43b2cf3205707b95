"""The transport's compiled variants against one another.

A queued run without reverse-path history, staged tables or records takes variants with
that code left out; `stage_tables` and `no_replay` select the general ones.  Both must give
the same tallies and counts: binary64 to 1e-12 of each sensor's largest bin (order of the
sums), binary32 to 1e-5 of it (separate compilations may round a binary32 operation
differently; every photon keeps its discrete history, so counts are equal).
"""
import numpy as np
import pytest

import luminis_mc_b200 as lm
from luminis_mc_b200 import workloads as W
from luminis_mc_b200.device import DeviceRun

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "fp32": 1e-5}


def _fluence_only(n):                 # no CBS sensor: nothing to replay
    spec = W.bilayer_rgd_mie(n, 3)
    spec["sensors"] = spec["sensors"][1:]
    return spec


def _statistics(n):                   # the penetration depth rides along
    spec = W.mie_cbs_small(n, 4)
    spec["sensors"].append({"kind": "statistics", "z": 0.0, "absorb": True, "events": 200,
                            "theta": [0.0, 1.6, 16], "depth": [2.0, 64]})
    return spec


def _mixture_absorption(n):
    spec = W.mixture_bilayer(n, 5)
    spec["absorption"] = {"radius": 5.0, "depth": 2.0, "d_r": 0.25, "d_z": 0.1}
    return spec


def run_tallies(spec, precision, **options):
    cfg, _, keep = W.build(lm, spec)
    run = DeviceRun(cfg)
    stats, _ = run.run(spec["n_photons"], spec["seed"], precision=precision, **options)
    out = [t.copy() for t in run.host_tallies()]
    grid = run.host_absorption()
    run.close()
    return stats, out + ([] if grid is None else [grid.copy()])


def assert_same_run(a, b, tol):
    (sa, ta), (sb, tb) = a, b
    for key in ("photons", "events", "steps", "draws", "hits", "detected", "escaped", "stack",
                "roulette", "cap", "error_flags"):
        assert sa[key] == sb[key], key
    assert len(ta) == len(tb)
    for x, y in zip(ta, tb):
        np.testing.assert_allclose(x, y, rtol=0, atol=tol * max(np.abs(y).max(), 1e-300))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [301, 19_001], ids=["short_run", "long_run"])
@pytest.mark.parametrize("make", [_fluence_only, _statistics, _mixture_absorption],
                         ids=["fluence_only", "statistics", "mixture_absorption"])
def test_variants_without_history_equal_the_general_ones(make, n, precision, cuda):
    """(runs of at most 128 photons per SM track the history instead of replaying)"""
    spec = make(n)
    default = run_tallies(spec, precision)
    assert default[0]["events"] > 0
    # (two blocks per SM: the kernels that count events per thread, not per block)
    for options in ({"stage_tables": True}, {"no_replay": True, "stage_tables": True},
                    {"blocks_per_sm": 2}, {"blocks_per_sm": 2, "no_replay": True}):
        assert_same_run(run_tallies(spec, precision, **options), default, TOL[precision])


def _depth(n, planes, absorb=False, absorption=False, cone=True):
    """Planes inside the sample beside the surface sensors: fluence at `planes` depths (one
    on the interface), statistics, a field grid; `absorb`: the deepest one ends photons."""
    spec = W.bilayer_rgd_mie(n, 6)
    spec["sensors"] = [spec["sensors"][0]]
    for i in range(planes):
        spec["sensors"].append({"kind": "planar_fluence", "z": 0.125 * (i + 1), "len_x": 4.0, "len_y": 4.0,
                                "len_t": 8.0, "dx": 0.25, "dy": 0.25, "d_t": 2.0,
                                "absorb": absorb and i == planes - 1})
    if planes < 5:
        spec["sensors"] += [{"kind": "statistics", "z": 0.25, "absorb": False, "events": 64,
                             "depth": [2.0, 16], "direction_limit": "backward"},
                            {"kind": "planar_field", "z": 0.3, "len_x": 2.0, "len_y": 2.0, "dx": 0.25,
                             "dy": 0.25, "absorb": False},
                            {"kind": "farfield_fluence", "theta_max": W.PI / 2, "phi_max": 2 * W.PI,
                             "len_t": 0.0, "d_theta": W.PI / 18, "d_phi": W.PI / 6, "d_t": 0.0}]
    if absorption:
        spec["absorption"] = {"radius": 3.0, "depth": 2.0, "d_r": 0.25, "d_z": 0.1}
    if not cone:
        spec["sensors"] = spec["sensors"][1:]
    return spec


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,planes,absorb,absorption,block,cone", [
    (7, 1, False, False, 0, False), (3001, 4, False, True, 0, False), (9001, 7, True, False, 64, False),
    (200_003, 4, True, False, 128, True), (200_003, 7, False, False, 0, True)])
def test_buffered_hits_equal_hits_on_the_spot(n, planes, absorb, absorption, block, cone, precision, cuda):
    """Scenes with planes inside the sample buffer their hits per warp and, in runs long
    enough, run the photons a CBS grid reads again; `no_replay` processes every hit on the
    spot.  The tallies, the counts and the Absorption grid are equal."""
    spec = _depth(n, planes, absorb, absorption, cone)
    a = run_tallies(spec, precision, block_size=block)
    b = run_tallies(spec, precision, no_replay=True)
    assert a[0]["replay_launches"] == (1 if cone else 0) and b[0]["replay_launches"] == 0
    assert_same_run(a, b, TOL[precision])
    assert_same_run(run_tallies(spec, precision, batch_photons=max(1, n // 3)), b, TOL[precision])


def _long(n):
    spec = W.mie_long_paths(n, 8)
    spec["max_events"] = 4000
    return spec


@pytest.mark.parametrize("make,n", [(W.mie_cbs_small, 1), (W.mie_cbs_small, 255), (W.mie_cbs_small, 257),
                                    (_long, 700), (W.bilayer_rgd_mie, 5003), (_mixture_absorption, 3001)])
@pytest.mark.parametrize("options", [{}, {"no_replay": True}, {"blocks_per_sm": 2}, {"blocks_per_sm": 1}],
                         ids=["default", "tracked", "two_blocks", "one_block"])
def test_packing_at_the_end_of_a_launch_changes_nothing(make, n, options, cuda):
    """Blocks of 8 warps pack their last photons into fewer warps; blocks of one warp have
    nothing to pack.  The same kernel computes the same photons: equal to the order of the
    tallies' sums."""
    spec = make(n, 8) if make in (W.mie_cbs_small, W.bilayer_rgd_mie) else make(n)
    packed = run_tallies(spec, "fp32", block_size=256, **options)
    assert_same_run(packed, run_tallies(spec, "fp32", block_size=32, **options), 1e-12)
    assert_same_run(packed, run_tallies(spec, "fp32", block_size=96, **options), 1e-12)


def test_packing_moves_records_and_scores(cuda):
    """Every per-photon record (reverse-path history included) and the likelihood-ratio
    scores survive the moves."""
    from luminis_mc_b200.adjoint import AdjointTransport
    spec = W.bilayer_rgd_mie(3000, 12)
    recs = []
    for block in (256, 32):
        cfg, _, keep = W.build(lm, spec)
        run = DeviceRun(cfg)
        recs.append(run.run(3000, 12, precision="fp32", records=True, block_size=block)[1])
        run.close()
    assert recs[0].tobytes() == recs[1].tobytes()
    # scores: two photon ranges of one launch size each against one launch
    cfg, _, keep = W.build(lm, W.bilayer_hg(4000, 13))
    tr = AdjointTransport(cfg, radial_sensor=1, radial_bins=20, radial_max=5.0)
    _, whole, _ = tr.run(4000, 13)
    parts = [tr.run(n, 13, begin=b)[1] * n for b, n in ((0, 31), (31, 1), (32, 3968))]
    tr.close()
    got, want = (sum(parts) / 4000).cpu().numpy(), whole.cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())


@pytest.mark.parametrize("n_div", [1, 2, 127, 1022, 1023, 1024, 2500])
def test_batched_cdf_at_chunk_edges(n_div, cuda):
    """The batched tables' CDF sums run in chunks of 1024 nodes: bit for bit the host's."""
    species = [(W.LAMBDA, r, W.N_SPHERE, W.N_WATER) for r in (0.05e-3, 0.4e-3, 2.0e-3)]
    for (ph, _), q in zip(lm.mie_species(species, n_div, 0.2, 2.9), species):
        ref = lm.MiePhaseFunction(*q, n_div, 0.2, 2.9)
        np.testing.assert_array_equal(ph._table()[1], ref._table()[1])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,bins", [(1, 40), (37, 100), (2500, 33)])
def test_spread_estimator_runs_equal_dense_ones(n, bins, precision, cuda):
    """Estimator runs with fewer photons than lanes spread them over all warps; one block per
    SM of one warp holds them densely.  Same estimates, other order of the sums."""
    spec = W.mie_cbs_small(n, 21)
    spec["sensors"] = [dict(spec["sensors"][0], estimator=True, d_theta=0.1 / bins)]
    spread = run_tallies(spec, precision)
    assert_same_run(spread, run_tallies(spec, precision, block_size=32, blocks_per_sm=1), 1e-12)


def test_first_run_of_a_scene_with_inner_planes_can_be_captured(cuda):
    """Under stream capture nothing may be allocated: a scene with inner planes whose buffers
    do not exist yet then processes its hits on the spot."""
    import torch
    spec = _depth(2000, 2, cone=False)
    stats, want = run_tallies(spec, "fp32", no_replay=True)
    cfg, _, keep = W.build(lm, spec)
    run = DeviceRun(cfg)
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        run.transport.run_device(run.tallies.data_ptr(), 2000, spec["seed"], want_stats=False,
                                 stream=stream.cuda_stream)
    for _ in range(2):
        run.zero()
        graph.replay()
        for x, y in zip(run.host_tallies(), want):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-12 * max(np.abs(y).max(), 1e-300))
    del graph
    run.close()
