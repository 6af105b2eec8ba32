"""The quasi-stationary kernels at the edges of their site sizes (one RyR, a full and a just
exceeded lane bitmask, the largest site whose increments sit in shared memory and the next), and
for each gating law they serve, against the restatement: identical event sequences and draw
counts, event times to 1e-12 (the tolerance of the other Gillespie tests)."""
import os

import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs
from oracle import qs_oracle

pytestmark = pytest.mark.gpu


def _run(p, coords, tmp_path, S=48, max_events=8192):
    np.savetxt(os.path.join(str(tmp_path), "coords.txt"), coords, fmt="%.17g")
    q = cb.QuasiStationarySites(p, S, base_dir=str(tmp_path), max_events=max_events)
    cfg = qs_oracle.parse(p, str(tmp_path))
    added = q.increments()
    seeds = qs_oracle.stream_seeds(S)
    first = ((np.arange(S) * 7) % q.n_ch).astype(np.int32)
    q.run(first)
    for s in range(S):
        t, c, st = q.events(s)
        to, co, so, d, _ = qs_oracle.run(cfg, added, seeds[s], int(first[s]))
        assert np.array_equal(c, co) and np.array_equal(st, so), s
        assert q.draws(s) == d
        if len(t):
            assert np.max(np.abs(t - to) / np.abs(to)) <= 1e-12, s
    q.close()


@pytest.mark.parametrize("n_ryr", [1, 3, 31, 32, 33, 64, 65, 70])
def test_site_sizes(cuda_device, tmp_path, n_ryr):
    p, coords = configs.quasi_stationary(n_ryr, seed=n_ryr, max_time=8.0)
    _run(p, coords, tmp_path)


@pytest.mark.parametrize("n_ryr", [5, 40])
def test_power_law(cuda_device, tmp_path, n_ryr):
    p, coords = configs.quasi_stationary(n_ryr, seed=2, max_time=8.0)
    ch = p["Calcium Release Site"]["Parameters"]["Channels"]["RyR"]
    ch["Model"] = "SheepCannell"
    ch["Parameters"] = configs.sheep_cannell_power_law()
    _run(p, coords, tmp_path)
