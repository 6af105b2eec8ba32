"""AUTO's choice for 3D dyads with the RD3D cytosol whose state the L2 holds: batches of few rounds
of the chip's clusters run resident, batches of many stream, and either way the results are those
of both paths: identical RyR states and draw counts, fields within the paths' common error (FP32
fields are each within 1e-5 of a species' largest value of the FP64 ones, so 2e-5 of one another;
FP64: 1e-11)."""
import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs

pytestmark = pytest.mark.gpu


def _batch(kind, n, side):
    if kind == "mg":
        return configs.config5(n_sites=2 * n, side=side)[0]
    return configs.config2(n_sites=n, side=side, ryr=(10, 100) if side[0] >= 40 else (3, 9))


@pytest.mark.parametrize("kind,precision,side,n,path", [("ca", "fp32", (40, 120), 33, "resident"), ("ca", "fp32", (40, 120), 65, "plain"),
                                                        ("ca", "fp32", (41, 60), 257, "plain"), ("ca", "fp64", (13, 30), 97, None),
                                                        ("mg", "fp32", (40, 57), 32, "resident"), ("mg", "fp32", (40, 57), 129, "plain")])
def test_auto_equals_both_paths(cuda_device, kind, precision, side, n, path):
    p, s = _batch(kind, n, side)
    got = {}
    for which in ("auto", "resident", "plain"):
        try:
            sim = cb.ReleaseSiteBatch(p, s, precision=precision, path=which)
        except cb.CasimError:  # sites that fit no cluster: AUTO streams them
            assert which == "resident" and auto == "plain"
            continue
        if which == "auto":
            auto = sim.path
        if which == "auto" and path:
            assert sim.path == path, sim.path_note()
        sim.start(s["first_channel"])
        sim.step(40)
        watch = (0, n // 2, n - 1)
        got[which] = (sim.all_states(), [sim.draws(k) for k in watch], [sim.field(k, f) for k in watch for f in range(sim.info.n_ions + sim.info.n_pairs)])
        sim.close()
    tol = 1e-11 if precision == "fp64" else 2e-5
    for which in set(got) - {"auto"}:
        assert np.array_equal(got["auto"][0], got[which][0])
        assert got["auto"][1] == got[which][1]
        for u, v in zip(got["auto"][2], got[which][2]):
            assert np.max(np.abs(u - v)) <= tol * np.max(np.abs(v))


def test_per_site_gating_is_refused_as_before(cuda_device):
    """A batch whose state the L2 holds takes per-site gating laws only on the plain path by name."""
    p, s = configs.config2(n_sites=65)
    sim = cb.ReleaseSiteBatch(p, s, precision="fp32", path="auto")
    assert sim.path == "plain"
    with pytest.raises(Exception, match="plain path"):
        sim.set_site_gating(p, [0])
    sim.close()
