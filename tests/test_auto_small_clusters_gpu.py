"""AUTO's choice for RD3D batches in L2 whose resident sites take one or two thread blocks, or another
grid than 25^3: resident where the streaming kernels measured slower, streaming from the seventh round of
clusters of four and more on. (The batches with the 25^3 grid are in the other AUTO test.)"""
import json
import re

import pytest

import casim_b200 as cb
from casim_b200 import configs

pytestmark = pytest.mark.gpu


def _batch(dim, ions, nodes, side, n):
    p, s = configs.config2(n_sites=n, seed=7, side=side, ryr=(5, 12) if side[0] < 40 else (10, 60))
    if dim == 2:
        p = configs._clean(configs.base_params(dim=2, cytosol="RD3D"))
        s["nz"] = s["nz"] * 0 + 1
    p = json.loads(json.dumps(p))
    if ions == 2:
        p = configs.with_magnesium(p)
    p["Cytosol"]["Nodes"] = nodes
    return p, s


@pytest.mark.parametrize("precision,dim,ions,nodes,side,n,path", [
    ("fp32", 3, 1, 9, (12, 24), 1500, "resident"), ("fp64", 3, 1, 9, (12, 24), 1500, "resident"), ("fp32", 2, 1, 9, (12, 24), 3000, "resident"),
    ("fp64", 3, 1, 16, (12, 24), 700, "resident"), ("fp32", 2, 2, 9, (40, 60), 1200, "resident"), ("fp64", 2, 1, 16, (40, 60), 400, "resident"),
    ("fp32", 2, 1, 25, (12, 14), 318, "resident"), ("fp64", 2, 1, 16, (100, 120), 75, "resident"), ("fp64", 2, 1, 16, (100, 120), 100, "plain"),
    ("fp32", 3, 2, 9, (60, 80), 141, "resident"), ("fp32", 3, 2, 9, (60, 80), 273, "plain"), ("fp64", 3, 1, 20, (40, 60), 100, "plain")])
def test_path(cuda_device, precision, dim, ions, nodes, side, n, path):
    p, s = _batch(dim, ions, nodes, side, n)
    sim = cb.ReleaseSiteBatch(p, s, precision=precision)
    assert sim.path == path, sim.path_note()
    sim.close()


def test_larger_clusters_by_name_stay_resident(cuda_device):
    p, s = _batch(3, 1, 9, (12, 24), 800)
    p["B200"] = {"MinClusterSize": 4}
    sim = cb.ReleaseSiteBatch(p, s, precision="fp32")
    assert sim.path == "resident" and set(re.findall(r"clusters of (\d+)", sim.path_note())) == {"4"}, sim.path_note()
    sim.close()
