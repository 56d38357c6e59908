"""Which domains of an ensemble are stepped together follows from what is still running,
after new targets as after a read (rb_ensemble_route)."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_ensemble_group import _member  # noqa: E402

# two members large enough for a group, and one that runs on when they have stopped
SIDES = {"local_inertial": [(1203, 1100), (811, 701), (300, 500)], "hllc_fv": [(1501, 1403), (1007, 1001), (230, 321)]}


@pytest.mark.parametrize("scheme", ["local_inertial", "hllc_fv"])
def test_new_targets_group_only_domains_that_still_run(scheme):
    from rbsim.ensemble import Ensemble
    from rbsim.scheduler import EPS_T

    hl = scheme == "hllc_fv"
    bit, unit = (2, 0.5) if hl else (1, 20.0)
    far = 100.0 * unit
    members = [_member(scheme, ny, nx, k, "plain") for k, (ny, nx) in enumerate(SIDES[scheme])]
    ens = Ensemble(members, [scheme] * 3, alpha=0.45 if hl else 0.7, dt_max=30.0, sync_times=[[unit], [unit], [far]],
                   graph_steps=2)  # fmt: skip

    def route():
        return ens._L.rb_ensemble_route(ens._ws.data_ptr())

    ens.set_targets([unit, unit, far])
    assert route() == bit
    for _ in range(1000):
        ens.replay()
        if all(c.t >= unit - EPS_T for c in ens.read()):
            break
    assert route() == 0 and ens.clock[2].t < far - EPS_T
    ens.set_targets([unit, unit, far])  # as the server does after an output frame
    assert route() == 0
    ens.set_targets([ens.clock[0].t + 0.5 * EPS_T, ens.clock[1].t + 0.5 * EPS_T, far])  # the clocks take no step to these
    assert route() == 0
    ens.set_targets([2.0 * unit, 2.0 * unit, far], max_steps=[0, 0, 10])
    assert route() == 0
    ens.set_targets([2.0 * unit, 2.0 * unit, far])  # the large ones run again
    assert route() == bit


@pytest.mark.parametrize("scheme", ["local_inertial", "hllc_fv"])
def test_autotune_times_the_work_list_with_every_member_on_it(scheme):
    """Its choice is of the work-list's tiles, which grouped members are not on."""
    from rbsim.ensemble import Ensemble, autotune

    hl = scheme == "hllc_fv"
    members = [_member(scheme, ny, nx, k, "plain") for k, (ny, nx) in enumerate(SIDES[scheme])]
    probes = []

    def make(li_v, hl_v, t0):
        e = Ensemble(members, [scheme] * 3, alpha=0.45 if hl else 0.7, dt_max=30.0, sync_times=[[1e6]] * 3,
                     li_variant=li_v, hllc_variant=hl_v, graph_steps=2, t0=0.0 if t0 is None else t0)  # fmt: skip
        e.set_targets(1e6)
        probes.append(e)
        return e

    (li_v, hl_v), timings, t0 = autotune(make, probe_replays=1, candidates=[(0, 0), (3, 2)])
    assert len(timings) == 2 and all(set(e._graphs) == {0} for e in probes)
    run = make(li_v, hl_v, t0)
    assert run._L.rb_ensemble_route(run._ws.data_ptr()) == (2 if hl else 1)
    run.allow_groups(False)
    run.set_targets(1e6)
    assert run._L.rb_ensemble_route(run._ws.data_ptr()) == 0
    run.allow_groups(True)
    run.read()
    assert run._L.rb_ensemble_route(run._ws.data_ptr()) == (2 if hl else 1)
