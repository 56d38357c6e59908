"""Ensembles whose larger members are stepped by one grouped launch of the row-streaming
kernels: every member equals its run alone bit for bit, while the group runs and after
its large members have stopped and the remaining ones are stepped by tiles again."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MM_H = 1.0 / 3.6e6
# Large members enough for a group, ragged in both directions; a wide one row, too flat for
# the strips' ledger slots; a middle one that runs on when the large ones have stopped; and
# small ones, more together than one launch holds (32).
SIDES = {
    "local_inertial": [(1203, 1100), (811, 701), (1, 300), (300, 500)] + [(33, 40 + k) for k in range(32)],
    "hllc_fv": [(1501, 1403), (1007, 1001), (2, 500), (230, 321)] + [(40, 61 + k) for k in range(32)],
}


def _member(scheme, ny, nx, seed, sources):
    import rbsim

    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:ny, 0:nx].astype(np.float64)
    dx = 10.0 if scheme == "local_inertial" else 2.0
    z = (1e-3 * x * dx + 0.2 * np.sin(y * 0.3) * np.cos(x * 0.2)).astype(np.float32)
    depth = np.maximum(rng.uniform(-0.1, 0.6, (ny, nx)), 0.0).astype(np.float32)
    if scheme == "hllc_fv":
        depth[:, : nx // 2] += 1.0
    st = rbsim.State.from_bed(z, dx, depth=depth, manning=0.03)
    if scheme == "hllc_fv":
        st.arm_hllc_fields()
    if sources == "mixed" and seed % 3 == 0:
        st.set_rain_field(torch.full((ny, nx), 40.0 * MM_H, device="cuda"))
        st.set_infiltration(torch.full((ny, nx), 2000.0 * MM_H, device="cuda"))
    if sources == "compensated" or (sources == "mixed" and seed % 2 == 0):
        st.arm_source_compensation()
    if seed % 2 == 0:
        st.set_open_boundaries({"east": "open", "north": "open"})
    return st


@pytest.mark.parametrize("sources", ["plain", "compensated", "mixed"])
@pytest.mark.parametrize("scheme", ["local_inertial", "hllc_fv"])
def test_grouped_members_equal_solo_runs(scheme, sources):
    from rbsim.device_clock import DeviceClock
    from rbsim.ensemble import Ensemble

    sides = SIDES[scheme]
    hl = scheme == "hllc_fv"
    alpha, bit = (0.45, 2) if hl else (0.7, 1)
    horizon = [(0.5 if hl else 20.0) * (3.0 if k == 3 else 1.0) for k in range(len(sides))]
    rain = 0.0 if sources == "plain" and hl else 50.0 * MM_H
    how = dict(dt_max=30.0, limit=True)
    solo = []
    for k, (ny, nx) in enumerate(sides):
        st = _member(scheme, ny, nx, k, sources)
        clk = DeviceClock(st, scheme, alpha=alpha, sync_times=[horizon[k]], rain_rate=rain, rain_until=horizon[k],
                          graph_steps=4, **how)  # fmt: skip
        clk.run_until(horizon[k])
        solo.append((st.h.cpu().numpy(), clk.steps, st.loss_cum.total() if st.loss_cum is not None else 0.0))
        clk.close()
    members = [_member(scheme, ny, nx, k, sources) for k, (ny, nx) in enumerate(sides)]
    ens = Ensemble(members, [scheme] * len(sides), alpha=alpha, sync_times=[[t] for t in horizon], rain_rate=rain,
                   rain_until=horizon, li_variant=3, hllc_variant=2, graph_steps=2, **how)  # fmt: skip
    ens.set_targets(horizon)
    route = ens._L.rb_ensemble_route
    assert route(ens._ws.data_ptr()) == bit
    ens.run_until(horizon)
    assert set(ens._graphs) == {bit, 0}  # grouped, then not
    for k, (st, (h, steps, loss)) in enumerate(zip(members, solo, strict=True)):
        assert ens.clock[k].steps == steps, k
        np.testing.assert_array_equal(st.h.cpu().numpy(), h, err_msg=f"member {k}")
        if loss:
            assert st.loss_cum.total() == pytest.approx(loss, rel=1e-12)
