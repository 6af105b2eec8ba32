"""The asynchronous streaming stencils (bulk copies into shared memory) at the sizes where
their tiling can go wrong, against the oracle over 120 steps: rows of 1 to 4 nodes of
padding, sites smaller and larger than a tile, a tile holding the first and the last row, odd
and even grids of the RD3D cytosol (25: planes through shared memory, others direct), batches
on both sides of the cytosol's split into chunks, the layouts that run the direct cleft kernel
(two ions and four pairs, FP64). FP64 1e-11 per node, identical RyR states and draws (the
tolerance of the other uneven-batch tests); FP32 1e-5 of each species' scale."""
import json

import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs
from oracle import oracle
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


def _sites(sides, dim, nodes=25, cytosol="RD3D", buffers=2, mg=False):
    n = len(sides)
    p, s = configs.small_mixed(n_sites=n, seed=3, dim=dim, cytosol=cytosol, side=(12, 13), ryr=(3, 4))
    s["nx"] = np.array([a for a, _ in sides], np.int32)
    s["ny"] = np.array([b for _, b in sides], np.int32)
    off = np.concatenate([[0], np.cumsum(s["n_ch"])])
    rng = np.random.default_rng(7)
    for k, (a, b) in enumerate(sides):
        s["ch_x"][off[k]:off[k + 1]] = rng.uniform(10.0, (a - 2) * 10.0, off[k + 1] - off[k])
        s["ch_y"][off[k]:off[k + 1]] = rng.uniform(10.0, (b - 2) * 10.0, off[k + 1] - off[k])
    if cytosol == "RD3D":
        p["Cytosol"]["Nodes"] = nodes
    if buffers > 2:
        for k in range(buffers - 2):
            p["Dyad"]["Buffers"]["Mobile%d" % k] = {"Total Concentration": 100.0 + k, "Ions": {"Calcium": {"D": 50000.0 * k, "kon": 0.05, "koff": 0.5}}}
    if mg:
        p = configs.with_magnesium(p)
        s["jsr_init"] = np.concatenate([s["jsr_init"], np.full((n, 1), 1000.0)], axis=1)
    return p, s


CASES = {
    "ragged3d": dict(sides=[(5, 5), (7, 40), (40, 7), (33, 34), (41, 23), (64, 8), (130, 12)], dim=3),
    "ragged2d": dict(sides=[(5, 5), (6, 200), (200, 6), (63, 65), (31, 17)], dim=2, cytosol="Pool"),
    "one_row_tiles": dict(sides=[(600, 7), (301, 9)], dim=2, cytosol="Pool"),
    "pool3d": dict(sides=[(21, 22), (50, 11)], dim=3, cytosol="Pool"),
    "even_cytosol": dict(sides=[(20, 21), (37, 30)], dim=3, nodes=12),
    "mg": dict(sides=[(18, 29), (35, 22)], dim=3, mg=True),
    "wide": dict(sides=[(22, 19), (27, 35)], dim=3, cytosol="Pool", buffers=4, mg=True),
}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_ragged_sites_match_oracle(cuda_device, case, precision):
    p, s = _sites(**CASES[case])
    _compare(p, s, precision, 120)


@pytest.mark.parametrize("n", [255, 256])
def test_cytosol_chunks_agree(cuda_device, n):
    """255 and 256 sites run the cytosol in three and two chunks: the first and last sites
    equal the same sites in a batch of two, bit for bit."""
    p, s = configs.config2(n_sites=n, seed=5, side=(12, 16), ryr=(2, 4))
    few = configs.subset_sites(s, [0, n - 1])
    sims = []
    for t in (s, few):
        sim = cb.ReleaseSiteBatch(p, t, precision="fp32", path="plain")
        sim.start(t["first_channel"])
        sim.step(50)
        sims.append(sim)
    for a, b in ((0, 0), (n - 1, 1)):
        for c in range(3):
            assert np.array_equal(sims[0].cyto_field(a, c), sims[1].cyto_field(b, c))
            assert np.array_equal(sims[0].field(a, c), sims[1].field(b, c))
    for sim in sims:
        sim.close()


def test_batches_of_different_rows_side_by_side(cuda_device):
    """Two handles whose tiles need different shared memory, stepped in turn: each equals its own
    run alone (the kernels' shared-memory cap is common to all handles)."""
    big, small = configs.config2(n_sites=3, seed=5, side=(110, 120), ryr=(4, 6)), configs.config2(n_sites=3, seed=6, side=(12, 16), ryr=(2, 4))
    alone = []
    for p, s in (big, small):
        sim = cb.ReleaseSiteBatch(p, s, precision="fp32", path="plain")
        sim.start(s["first_channel"])
        sim.step(20)
        alone.append([sim.field(k, 0) for k in range(3)])
        sim.close()
    sims = [cb.ReleaseSiteBatch(p, s, precision="fp32", path="plain") for p, s in (big, small)]
    for sim, (_, s) in zip(sims, (big, small)):
        sim.start(s["first_channel"])
    for _ in range(2):
        for sim in sims:
            sim.step(10)
    for sim, want in zip(sims, alone):
        for k in range(3):
            assert np.array_equal(sim.field(k, 0), want[k])
        sim.close()


def _compare(p, s, precision, steps):
    sim = cb.ReleaseSiteBatch(json.loads(json.dumps(p)), s, precision=precision, path="plain")
    orc = oracle.OracleSim(p, s)
    sim.start(s["first_channel"])
    orc.start(s["first_channel"])
    sim.step(steps)
    orc.step(steps)
    sim.synchronize()
    species = sim.info.n_ions + sim.info.n_pairs
    for k in range(sim.S):
        if precision == "fp64":
            assert np.array_equal(sim.states(k), orc.states(k)) and sim.draws(k) == orc.draws(k), k
        for sp in range(species):
            a, b = sim.field(k, sp), orc.field(k, sp)
            assert (rel_err(a, b) <= 1e-11) if precision == "fp64" else (np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(b))), (k, sp)
        for sp in range(sim.info.n_cyto_species if sim.info.cyto_nodes else 0):
            a, b = sim.cyto_field(k, sp), orc.cyto_field(k, sp)
            assert (rel_err(a, b) <= 1e-11) if precision == "fp64" else (np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(b))), (k, sp)
        assert rel_err(sim.jsr(k)[:1], orc.jsr(k)[:1]) <= (1e-12 if precision == "fp64" else 1e-5)
        if not sim.info.cyto_nodes:
            assert rel_err(sim.cyto(k), orc.cyto(k)) <= (1e-12 if precision == "fp64" else 1e-5)
    sim.close()
