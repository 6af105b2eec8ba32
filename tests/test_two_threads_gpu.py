"""Two threads, each stepping a batch of its own whose sites need another amount of shared memory in the
same kernels, as long as the other does: no launch fails, and each batch ends as it does alone.
(The cap on a kernel's shared memory is common to the process.)"""
import threading

import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs

pytestmark = pytest.mark.gpu


def _batch(side, path):
    p, s = configs.config2(n_sites=3, seed=side, side=(side, side), ryr=(10, 20))
    if path == "resident":
        p["Cytosol"]["Nodes"] = 9
    return p, s


@pytest.mark.parametrize("path,sides,steps", [("plain", (240, 320), 400), ("resident", (20, 32), 600)])
def test_two_batches_in_two_threads(cuda_device, path, sides, steps):
    want, sims = [], []
    for side in sides:
        p, s = _batch(side, path)
        for both in (want, sims):
            sim = cb.ReleaseSiteBatch(p, s, precision="fp32", path=path)
            sim.start(s["first_channel"])
            both.append(sim)
    for sim in want:
        for _ in range(steps):
            sim.step(1)
        sim.synchronize()
    errors = []
    go = threading.Barrier(2)

    def run(sim):
        try:
            go.wait()
            for _ in range(steps):
                sim.step(1)
            sim.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=run, args=(sim,)) for sim in sims]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for a, b in zip(want, sims):
        assert np.array_equal(a.all_states(), b.all_states())
        assert np.array_equal(a.field(1, 0), b.field(1, 0)) and np.array_equal(a.cyto_field(1, 0), b.cyto_field(1, 0))
        a.close()
        b.close()
