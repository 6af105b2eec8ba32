"""An infinite opening rate (a tetrameric law with nothing between the open and the closed conformation,
no Mg) in the quasi-stationary kernels: every share of the infinite total is zero or undefined, so
the reference's walk over the shares picks no RyR and takes RyR 0. Started from RyR 0 it closes at
once, as in the restatement: one event, at time zero."""
import os

import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs
from oracle import qs_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ryr", [2, 20, 33, 70])
def test_infinite_total(cuda_device, tmp_path, n_ryr):
    p, coords = configs.quasi_stationary(n_ryr, seed=n_ryr, max_time=2.0)
    par = p["Calcium Release Site"]["Parameters"]
    par["Channels"]["RyR"]["Parameters"]["KO0"] = 0.0
    par["Dyadic Cleft"]["Ions"]["Magnesium"]["Concentration"] = 0.0
    np.savetxt(os.path.join(str(tmp_path), "coords.txt"), coords, fmt="%.17g")
    S = 40
    q = cb.QuasiStationarySites(p, S, base_dir=str(tmp_path), max_events=4096)
    q.run(np.zeros(S, np.int32))
    cfg = qs_oracle.parse(p, str(tmp_path))
    seeds = qs_oracle.stream_seeds(S)
    for s in range(S):
        t, c, st = q.events(s)
        to, co, so, d, _ = qs_oracle.run(cfg, q.increments(), seeds[s], 0)
        assert np.array_equal(c, co) and np.array_equal(st, so) and np.array_equal(t, to), s
        assert q.draws(s) == d
    q.close()
