"""A batch whose kernel gave up a bounded wait (marked from the host: no wait fails here): every call
that reads its state, or would step it further, returns ETIMEOUT; start, or reset with its opening
and Update, makes it valid again, with the results of a batch that never failed."""
import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs

pytestmark = pytest.mark.gpu


def _timeouts(calls):
    for name, f in calls:
        with pytest.raises(cb.CasimError) as e:
            f()
        assert e.value.status == cb.ETIMEOUT, name


def _results(sim, rd3d):
    out = [sim.all_states(), sim.all_mouth(0), sim.jsr(1), np.array([sim.draws(1), sim.release(1)])]
    out += [sim.field(1, f) for f in range(sim.info.n_ions + sim.info.n_pairs)]
    return out + ([sim.cyto_field(1, 0)] if rd3d else [sim.cyto(1)])


@pytest.mark.parametrize("path,cytosol", [("plain", "RD3D"), ("plain", "Pool"), ("resident", "RD3D"), ("resident", "Pool")])
def test_reads_refuse_and_start_recovers(cuda_device, path, cytosol):
    rd3d = cytosol == "RD3D"
    p, s = configs.small_mixed(n_sites=3, dim=3, cytosol=cytosol)
    first = s["first_channel"]

    def fresh():
        sim = cb.ReleaseSiteBatch(p, s, path=path)
        sim.start(first)
        sim.trace_enable(10, 8)
        sim.step(30)
        return sim

    good, sim = fresh(), fresh()
    assert cb.lib().casim_b200_debug_give_up(sim.h) == cb.OK
    calls = [("step", lambda: sim.step(1)), ("synchronize", sim.synchronize), ("all_states", sim.all_states),
             ("all_mouth", lambda: sim.all_mouth(0)), ("field", lambda: sim.field(0, 0)), ("mouth", lambda: sim.mouth(0, 0)),
             ("states", lambda: sim.states(0)), ("jsr", lambda: sim.jsr(0)), ("efflux", lambda: sim.efflux(0)),
             ("total_current", lambda: sim.total_current(0)), ("draws", lambda: sim.draws(0)), ("release", lambda: sim.release(0)),
             ("cyto", lambda: sim.cyto(0)), ("open_traces", sim.open_traces), ("analysis", lambda: sim.release_analysis(0.001, 2)),
             ("trace_enable", lambda: sim.trace_enable(10, 8))]
    if rd3d:
        calls.append(("cyto_field", lambda: sim.cyto_field(0, 0)))
    _timeouts(calls)
    ok, bad = sim.check_finite()
    assert not ok and bad == -1
    # the streams have moved on in both, as on a second start of any batch
    good.start(first)
    good.step(20)
    sim.start(first)
    sim.step(20)
    for a, b in zip(_results(good, rd3d), _results(sim, rd3d)):
        assert np.array_equal(a, b)
    assert cb.lib().casim_b200_debug_give_up(sim.h) == cb.OK
    for b in (good, sim):
        b.reset()
        b.step(5)  # queued behind the reset: not refused
        b.reset()
        for k in range(3):
            b.init_opening(k, int(first[k]))
        b.update()
        b.step(10)
    for a, b in zip(_results(good, rd3d), _results(sim, rd3d)):
        assert np.array_equal(a, b)
    good.close()
    sim.close()


def test_profile_step_refuses(cuda_device):
    p, s = configs.small_mixed(n_sites=2, dim=3, cytosol="RD3D")
    sim = cb.ReleaseSiteBatch(p, s, path="plain")
    sim.start(s["first_channel"])
    assert cb.lib().casim_b200_debug_give_up(sim.h) == cb.OK
    _timeouts([("profile_step", sim.profile_step)])
    sim.start(s["first_channel"])
    assert sim.profile_step()["update"] > 0
    sim.close()


def test_surrogate_run_refuses(cuda_device):
    from casim_b200 import surrogate as sg
    p, s = configs.config1(n_sites=3)
    sim = cb.ReleaseSiteBatch(p, s, precision="fp32")
    net = sg.Surrogate(63, 20, width=64, depth=1)
    gate = sg.SurrogateGating(net, sim)
    sim.start(s["first_channel"])
    gate.step(40)
    assert cb.lib().casim_b200_debug_give_up(sim.h) == cb.OK
    _timeouts([("sg_run", lambda: gate.step(40)), ("hybrid", lambda: gate.hybrid_step(40))])
    sim.start(s["first_channel"])
    gate.step(40)
    sim.close()
    net.close()
