"""Azimuth rejection in binary32: the trials read straight from the photon's ring.

A binary32 event takes its trials from the numbers already in the ring (3 to 7 of them)
and continues draw by draw when they run out.  Particles much smaller than the wavelength
in linearly polarised light reject most often, so that both ways are taken; every photon
must consume exactly the oracle's draws.  Binary32 rounding (1e-7 of F) decides a trial
differently from binary64 with a probability of ~1e-7 per trial, i.e. for ~0.1 of the
photons of a run here: at most 2 of 2000 may differ.
"""
import numpy as np
import pytest

import luminis_mc_b200 as lm
from luminis_mc_b200 import workloads as W
from luminis_mc_b200.device import DeviceRun
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def _spec(radius, polarisation, n, seed):
    spec = W.mie_cbs_small(n, seed)
    spec["name"] = f"azimuth_{radius}_{polarisation}"
    spec["laser"] = W._laser(*(W.LINEAR if polarisation == "linear" else W.CIRCULAR))
    for table in (spec["phases"][0], spec["media"][0]):
        table["radius"] = radius
    spec["media"][0]["mu_a"] = 0.3
    return spec


@pytest.mark.parametrize("radius,polarisation", [(0.02e-3, "linear"), (0.02e-3, "circular"),
                                                 (1.0e-3, "linear")])
def test_binary32_trials_consume_the_oracles_draws(radius, polarisation, cuda):
    n, seed = 2000, 4711
    spec = _spec(radius, polarisation, n, seed)
    cfg, _, keep = W.build(lm, spec)
    run = DeviceRun(cfg)
    stats, rec = run.run(n, seed, precision="fp32", records=True)
    run.close()
    ref = O.Oracle(spec).run(n, seed, rng="philox_u24", records=True).records
    assert stats["error_flags"] == 0
    # two draws per event and two per trial, one trial at least: rejections must occur
    assert ref["draws"].sum() > 4.0 * ref["events"].sum()
    differ = ((rec["draws"] != ref["draws"]) | (rec["events"] != ref["events"]) |
              (rec["fate"] != ref["fate"]))
    assert np.count_nonzero(differ) <= 2
