"""RD3D cytosols of other grids than the shipped 25^3 in the streaming stencil, whose blocks, nodes per
thread and planes loaded ahead go by precision and species: the smallest grid, layers of a few nodes,
of just under and just over a block, and of several, even and odd rows, one to six species; against the
oracle over 40 steps with the tolerances of the other streaming tests (FP64 1e-11 per node and identical
RyR states and draws, FP32 1e-5 of each species' scale)."""
import json

import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs
from oracle import oracle
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


def _params(nodes, mg, extra):
    p, s = configs.small_mixed(n_sites=2, seed=nodes, dim=3, cytosol="RD3D", side=(12, 20), ryr=(3, 6))
    p = json.loads(json.dumps(p))
    p["Cytosol"]["Nodes"] = nodes
    for k in range(extra):
        p["Cytosol"]["Buffers"]["Y%d" % k] = {"Total Concentration": 30.0 + k, "Ions": {"Calcium": {"D": 2e4 * k, "kon": 0.08, "koff": 0.9}}}
    if mg:
        p = configs.with_magnesium(p)
        s["jsr_init"] = np.concatenate([s["jsr_init"], np.full((2, 1), 1000.0)], axis=1)
    return p, s


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nodes,mg,extra", [(4, False, 0), (5, True, 0), (8, False, 2), (11, False, 0), (12, True, 2), (15, False, 1), (16, True, 1),
                                            (23, False, 0), (26, True, 0), (27, False, 2), (30, True, 2), (37, False, 0)])
def test_grid_matches_oracle(cuda_device, nodes, mg, extra, precision):
    p, s = _params(nodes, mg, extra)
    sim = cb.ReleaseSiteBatch(p, s, precision=precision, path="plain")
    orc = oracle.OracleSim(p, s)
    for b in (sim, orc):
        b.start(s["first_channel"])
        b.step(40)
    sim.synchronize()
    for k in range(2):
        if precision == "fp64":
            assert np.array_equal(sim.states(k), orc.states(k)) and sim.draws(k) == orc.draws(k)
        pairs = [(sim.cyto_field(k, c), orc.cyto_field(k, c)) for c in range(sim.info.n_cyto_species)]
        pairs += [(sim.field(k, f), orc.field(k, f)) for f in range(sim.info.n_ions + sim.info.n_pairs)]
        for i, (a, b) in enumerate(pairs):
            assert (rel_err(a, b) <= 1e-11) if precision == "fp64" else (np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(b))), (k, i)
    sim.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_shipped_grid_with_six_species(cuda_device, precision):
    """25^3 with two ions and four pairs: as many species as the bulk copies' stages are counted for."""
    test_grid_matches_oracle(cuda_device, 25, True, 2, precision)
