"""The warp-parallel 60-state gating kernel at the edges of its 32-RyR chunks against the
oracle: identical micro-states and draw counts (every draw is the same bit for bit, so the
last draw of a chunk, its second draw and the stream state left behind all show), fields to
1e-11 (the FP64 tolerance of the other 60-state test)."""
import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs
from oracle import oracle
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ryr", [1, 31, 32, 33, 64, 70])
def test_sixty_state_chunks_match_oracle(cuda_device, n_ryr):
    params, sites = configs.config1(n_sites=3, seed0=40 + n_ryr, nx=32, ny=33, n_ryr=n_ryr)
    sites["ch_x"] = np.clip(sites["ch_x"], 20.0, 290.0)
    sites["ch_y"] = np.clip(sites["ch_y"], 20.0, 300.0)
    params = configs.with_single_site_mwc(params, speed=200.0)
    params["dt, ns"] = 10.0
    sim = cb.ReleaseSiteBatch(params, sites, precision="fp64", path="auto")
    orc = oracle.OracleSim(params, sites)
    sim.start(sites["first_channel"])
    orc.start(sites["first_channel"])
    moved = 0
    for chunk in (1, 60, 139):
        before = [orc.micro_states(s) for s in range(3)]
        sim.step(chunk)
        orc.step(chunk)
        for s in range(3):
            assert np.array_equal(sim.micro_states(s), orc.micro_states(s)), (chunk, s)
            assert np.array_equal(sim.states(s), orc.states(s))
            assert sim.draws(s) == orc.draws(s)
            assert rel_err(sim.field(s, 0), orc.field(s, 0)) <= 1e-11
            moved += int(np.sum(before[s] != orc.micro_states(s)))
    assert moved >= 2 * n_ryr
    sim.close()
