"""What a user of rbsim has the GPU do, as cases that can be timed and checked.

A case is one scenario and the way its program steps it:

* ``api = "step"``: the scheme loop, ``compute_dt`` then ``step`` for every step (the
  interface of the reference, which reads dt back to the host each time);
* ``api = "clock"``: ``DeviceClock.run_until``, what ``rbsim.run`` steps a scenario with;
* ``api = "ensemble"``: one ``Ensemble`` over many domains, what the server steps its
  requests with.

``prepare`` builds the states the program holds (inputs made on the GPU from the seed),
``run`` advances them by ``steps`` steps and returns the fields they then hold, and
``exact`` is the same advance in float64 with plain torch operations. A second ``run``
goes on from where the first one stopped, as a time loop does.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "river-basin-sim_b200"))

import rbsim  # noqa: E402
from rbsim import arith  # noqa: E402
from rbsim.channels import arm_channels  # noqa: E402
from rbsim.device_clock import DeviceClock  # noqa: E402
from rbsim.ensemble import Ensemble, log_uniform_sides  # noqa: E402
from rbsim.processes.inflow import Inflow, InflowInjector  # noqa: E402
from rbsim.sediment import arm_sediment  # noqa: E402

G, H_DRY = 9.81, 1e-3
RAIN = 50.0 / 3.6e6  # 50 mm/h
HORIZON = 1.0e9  # the run goes on past every pass
ALPHA = {"local_inertial": 0.7, "hllc_fv": 0.45}
DT_MAX = 30.0
EDGES = ("north", "south", "east", "west")


def listed() -> list[dict]:
    li, hl = "local_inertial", "hllc_fv"
    return [
        # an interactive step of a small catchment: launches and the dt read-back are all of it
        _case("li_step_97x161", li, 97, 161, 10.0, "step", "exact", 1, terrain="hills", edges="open", rain="uniform"),
        # the rain-on-grid configuration of the benchmark (512^2, 50 mm/h, open edges)
        _case("li_rain_512", li, 512, 512, 10.0, "clock", "exact", 32, terrain="hills", edges="open", rain="uniform"),
        # the same, as large as a county-wide 10 m model, in the arithmetic a throughput run picks
        _case("li_rain_2048_fast", li, 2048, 2048, 10.0, "clock", "fast", 32, terrain="hills", edges="open",
              rain="uniform"),
        # a radar rain field over soils that infiltrate, on a ragged grid cut from a mosaic
        _case("li_field_1531x1017", li, 1531, 1017, 10.0, "clock", "exact", 32, terrain="hills", edges="open",
              rain="field", infil=True),
        # the scheme loop on a large grid: what a program ported from the reference runs
        _case("li_step_2048", li, 2048, 2048, 10.0, "step", "exact", 4, terrain="hills", edges="closed",
              rain="uniform"),
        # the valley reach of the benchmark: inflows, infiltration and bedload, the largest domain
        _case("li_reach_8192_fast", li, 8192, 8192, 5.0, "clock", "fast", 8, terrain="valley", edges="east",
              infil=True, sediment=True, inflows=8),
        # the reference's alluvial reach: 768^2 at 100 m with sub-grid channels and bedload
        _case("li_channels_768", li, 768, 768, 100.0, "clock", "exact", 32, terrain="valley", edges="east",
              sediment=True, channels=True, inflows=4),
        # a small dam break
        _case("hllc_dam_256", hl, 256, 256, 1.0, "clock", "exact", 32, terrain="dam", edges="closed"),
        # the headline configuration of the benchmark
        _case("hllc_dam_2048_fast", hl, 2048, 2048, 1.0, "clock", "fast", 32, terrain="dam", edges="closed"),
        # waves over submerged and emergent bumps with friction: the wet / dry branches
        _case("hllc_lake_2048", hl, 2048, 2048, 1.0, "clock", "exact", 16, terrain="lake", edges="closed"),
        # a storm over a coast: rain field, infiltration, open edges and a sea level, ragged, scheme loop
        _case("hllc_storm_1013x757", hl, 1013, 757, 2.0, "step", "exact", 4, terrain="lake", edges="stage",
              rain="field", infil=True),
        # a batch of requests of both schemes
        dict(name="ensemble_20", scheme="mixed", api="ensemble", arith="exact", domains=20, lo=128, hi=1400, steps=8,
             layout_seed=7, li_variant=3, hllc_variant=2),
    ]  # fmt: skip


def _case(name, scheme, ny, nx, dx, api, arithmetic, steps, **more) -> dict:
    c = dict(scheme=scheme, ny=ny, nx=nx, dx=dx, api=api, arith=arithmetic, steps=steps, terrain="hills",
             edges="closed", rain="none", infil=False, sediment=False, channels=False, inflows=0)  # fmt: skip
    c.update(more)
    return dict(c, name=name) if name else c


def draw(rng) -> dict:
    """A scenario of the same ranges: either scheme, any stepping, odd sizes and long
    sides among them, the options that the run configurations arm."""
    kind = rng.choice(("li", "li", "reach", "hllc", "hllc", "ensemble"))
    if kind == "ensemble":
        return dict(scheme="mixed", api="ensemble", arith="exact", domains=rng.randint(3, 20), lo=rng.randint(64, 256),
                    hi=rng.randint(300, 1400), steps=rng.choice((4, 8, 16)), layout_seed=rng.randrange(1 << 20),
                    li_variant=rng.choice((0, 3)), hllc_variant=rng.choice((0, 2)))  # fmt: skip
    side = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    api, mode = rng.choice(("clock", "clock", "step")), rng.choice(("exact", "fast"))
    steps = rng.choice((1, 2, 4)) if api == "step" else rng.choice((8, 32))
    edges = rng.choice(("closed", "open", "east"))
    rain = rng.choice(("none", "uniform", "uniform", "field"))
    infil = rng.random() < 0.4
    if kind == "hllc":
        return _case(None, "hllc_fv", side(40, 2600), side(40, 2600), rng.choice((1.0, 2.0, 5.0)), api, mode, steps,
                     terrain=rng.choice(("dam", "lake")), edges=rng.choice((edges, "stage")), rain=rain,
                     infil=infil)  # fmt: skip
    if kind == "li":
        return _case(None, "local_inertial", side(40, 4000), side(40, 4000), rng.choice((5.0, 10.0, 30.0)), api, mode,
                     steps, terrain="hills", edges=edges, rain=rain, infil=infil)  # fmt: skip
    chan = rng.random() < 0.4
    return _case(None, "local_inertial", side(200, 3000), side(200, 3000), 100.0 if chan else rng.choice((5.0, 10.0)),
                 api, mode, steps, terrain="valley", edges="east", rain=rain, infil=infil,
                 sediment=rng.random() < 0.7, channels=chan, inflows=rng.randint(1, 8))  # fmt: skip


# --- inputs ------------------------------------------------------------------------


def _bumps(ny, nx, dx, gen, count, amp, sigma):
    """A sum of Gaussian bumps, each a product of a row and a column profile."""
    u = torch.rand(4, count, generator=gen, device="cuda", dtype=torch.float64)
    a = amp[0] + (amp[1] - amp[0]) * u[0]
    s = sigma[0] + (sigma[1] - sigma[0]) * u[1]
    y = torch.arange(ny, device="cuda", dtype=torch.float64)[:, None]
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None]
    gy = torch.exp(-(((y - u[2] * ny) * dx) ** 2) / (2 * s * s)) * a
    gx = torch.exp(-(((x - u[3] * nx) * dx) ** 2) / (2 * s * s))
    return (gy @ gx.T).float()


def _inputs(c: dict, seed: int) -> dict:
    """Everything the scenario is made of, float32 on the GPU."""
    ny, nx, dx = c["ny"], c["nx"], c["dx"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    rnd = lambda: torch.rand(ny, nx, generator=gen, device="cuda")  # noqa: E731
    col = torch.arange(nx, device="cuda", dtype=torch.float32)[None, :]
    row = torch.arange(ny, device="cuda", dtype=torch.float32)[:, None]
    ext = math.sqrt(ny * nx) * dx
    d = {"manning": 0.03}
    if c["terrain"] == "hills":
        d["bed"] = (1e-3 * col * dx + _bumps(ny, nx, dx, gen, 40, (0.5, 5.0), (0.02 * ext, 0.08 * ext))).contiguous()
        d["depth"] = 0.5 + 0.1 * rnd()
    elif c["terrain"] == "valley":
        phase = 6.28 * float(torch.rand(1, generator=gen, device="cuda"))
        centre = 0.5 * ny + 0.1 * ny * torch.sin(6.28 * col * dx / 3000.0 * (5.0 / dx) + phase)
        dist = (row - centre).abs() * dx
        chan = dist <= 4.0 * dx
        z = 0.005 * dist * (5.0 / dx) + 1e-3 * (nx - 1 - col) * dx
        d["bed"] = (torch.where(chan, z - 3.0, z) if not c["channels"] else z).contiguous()
        d["depth"] = torch.where(chan, torch.full_like(z, 2.0), torch.full_like(z, 0.05))
        d["manning"] = torch.exp(math.log(0.035) + 0.3 * torch.randn(ny, nx, generator=gen, device="cuda"))
        rows = torch.nonzero(chan[:, 0]).flatten()[: c["inflows"]].tolist()
        hydro = [(0.0, 0.0), (7200.0, 500.0 / max(len(rows), 1)), (14400.0, 0.0)]
        d["inflows"] = [((int(r), 0), hydro) for r in rows]
        if c["channels"]:  # a main stem narrower than its cell along the thalweg
            stem = dist <= 0.5 * dx
            d["chan_w"] = torch.where(stem, 0.2 * dx + 0.3 * dx * rnd(), torch.zeros_like(z))
            d["chan_d"] = torch.where(stem, 1.5 + rnd(), torch.zeros_like(z))
            d["depth"] = torch.where(stem, 0.8 * rnd() + 0.2, 0.05 * torch.ones_like(z))
    elif c["terrain"] == "dam":
        split = 0.3 + 0.4 * float(torch.rand(1, generator=gen, device="cuda"))
        d["bed"] = torch.zeros(ny, nx, device="cuda")
        line = col + 0.5 * row - 0.25 * ny  # a dam across the domain at an angle
        d["depth"] = (torch.where(line < split * nx, 10.0, 1.0) + 0.01 * rnd()).contiguous()
        d["manning"] = 0.0
    else:  # lake: a 2 m surface with waves on it over bumps, some of which pierce it
        d["bed"] = _bumps(ny, nx, dx, gen, 40, (0.2, 2.6), (0.01 * ext, 0.05 * ext))
        d["depth"] = torch.clamp(2.0 + _bumps(ny, nx, dx, gen, 8, (0.2, 0.6), (0.02 * ext, 0.06 * ext)) - d["bed"], min=0.0)
        d["depth"] = torch.where(d["depth"] < 5e-3, torch.zeros_like(d["depth"]), d["depth"])
        d["velocity"] = 0.5 * (2.0 * torch.rand(2, generator=gen, device="cuda") - 1.0)
    if c["rain"] == "field":
        d["rain_field"] = RAIN * 2.0 * rnd()
    if c["infil"]:
        d["infil"] = rnd() * (20.0 / 3.6e6)
    if c["edges"] != "closed":
        kinds = {"open": {e: "open" for e in EDGES}, "east": {"east": "open"},
                 "stage": {"west": "open", "north": "open", "east": "fixed_stage"}}[c["edges"]]  # fmt: skip
        d["boundaries"] = kinds
        # a sea level 0.3 m over the still water, falling as a tide does
        d["stage"] = {"east": [(0.0, 2.3), (36000.0, 1.7)]} if "fixed_stage" in kinds.values() else None
    return d


def _state(c: dict, d: dict):
    st = rbsim.State.from_bed(d["bed"], c["dx"], depth=d["depth"], manning=d["manning"])
    if c["scheme"] == "hllc_fv":
        st.arm_hllc_fields()
        if "velocity" in d:
            st.hu, st.hv = d["depth"] * d["velocity"][0], d["depth"] * d["velocity"][1]
    if "infil" in d:
        st.set_infiltration(d["infil"])
    if "rain_field" in d:
        st.set_rain_field(d["rain_field"])
    if c["rain"] != "none":
        st.arm_source_compensation()
    if "boundaries" in d:
        st.set_open_boundaries(d["boundaries"], d["stage"])
    if c["channels"]:
        w, dep = d["chan_w"].cpu().numpy(), d["chan_d"].cpu().numpy()
        arm_channels(st, w, dep, np.full_like(w, 0.03))
    if c["sediment"]:
        arm_sediment(st, 0.002, 0.4)
    return st


def _members(c: dict) -> list[dict]:
    """The domains of an ensemble: both schemes, sides log-uniform, as the server's mix."""
    sides = log_uniform_sides(c["domains"], c["lo"], c["hi"], c["layout_seed"])
    out = []
    for k, side in enumerate(sides):
        hl = k % 10 in (3, 6, 9)  # 70 % local inertial, 30 % HLLC
        out.append(_case(None, "hllc_fv" if hl else "local_inertial", side, max(32, side - 3 * (k % 5)),
                         2.0 if hl else 10.0, "clock", "exact", c["steps"], terrain="lake" if hl else "hills",
                         rain="none" if hl else "uniform"))  # fmt: skip
    return out


def prepare(case: dict, seed: int):
    c = dict(case)
    if c["api"] == "ensemble":
        members = _members(c)
        states = [_state(m, _inputs(m, seed * 1000 + k)) for k, m in enumerate(members)]
        ens = Ensemble(states, [m["scheme"] for m in members], alpha=[ALPHA[m["scheme"]] for m in members],
                       dt_max=DT_MAX, rain_rate=[RAIN if m["rain"] != "none" else 0.0 for m in members],
                       rain_until=HORIZON, li_variant=c["li_variant"], hllc_variant=c["hllc_variant"],
                       graph_steps=c["steps"])  # fmt: skip
        return {"case": c, "states": states, "ensemble": ens}
    d = _inputs(c, seed)
    st = _state(c, d)
    s = {"case": c, "state": st, "t": 0.0, "injector": None}
    if d.get("inflows"):
        s["injector"] = InflowInjector([Inflow(cell, h) for cell, h in d["inflows"]], st.grid, st.device)
    if c["api"] == "clock":
        s["clock"] = DeviceClock(st, c["scheme"], alpha=ALPHA[c["scheme"]], dt_max=DT_MAX, sync_times=[HORIZON],
                                 rain_rate=RAIN if c["rain"] == "uniform" else 0.0, rain_until=HORIZON,
                                 injector=s["injector"])  # fmt: skip
    return s


# --- one pass ------------------------------------------------------------------------


def _fields(st) -> dict:
    if st.hllc:
        return {"h": st.h, "hu": st.hu, "hv": st.hv}
    out = {"h": st.h, "qx": st.qx, "qy": st.qy}
    if st.channels is not None:
        out.update({k: getattr(st.channels, k) for k in ("qx_ch", "qx_fp", "qy_ch", "qy_fp")})
    if st.sediment is not None:
        out["qs_int_x"], out["qs_int_y"] = st.sediment.qs_int_x, st.sediment.qs_int_y
    return out


def run(state):
    c = state["case"]
    if c["api"] == "ensemble":
        ens = state["ensemble"]
        ens.set_targets(HORIZON)
        ens.replay()
        ens.read()
        return [_fields(st) for st in state["states"]]
    st = state["state"]
    with arith.using(c["arith"]):
        if c["api"] == "clock":
            state["clock"].run_until(HORIZON, max_steps=c["steps"])
        else:
            scheme, inj = rbsim.get_scheme(c["scheme"]), state["injector"]
            rain = RAIN if c["rain"] == "uniform" else 0.0
            for _ in range(c["steps"]):
                dt = scheme.compute_dt(st, alpha=ALPHA[c["scheme"]], dt_max=DT_MAX)
                if inj is not None:
                    inj.apply(st, state["t"], dt)
                scheme.step(st, dt=dt, rain=rain, t=state["t"])
                state["t"] += dt
    return _fields(st)


def work(case: dict) -> dict:
    """Per cell and step: every field the step needs read once and every one it changes
    written once (float32), and the arithmetic of its faces and its update."""
    if case["api"] == "ensemble":
        parts = [work(m) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    c = case
    per, flops = 32, 60  # h, z, n, qx, qy in and h, qx, qy out; h, hu, hv, z, n in and h, hu, hv out
    if c["scheme"] == "hllc_fv":
        flops = 2 * 2 * 100 + 2 * 40  # two stages of two faces and one update
    per += 8 * (c["rain"] != "none") + 4 * (c["rain"] == "field") + 4 * c["infil"]
    per += 36 * c["sediment"] + 44 * c["channels"]
    flops += 40 * c["sediment"] + 60 * c["channels"]
    n = c["ny"] * c["nx"] * c["steps"]
    return {"bytes": float(per * n), "flops": float(flops * n)}


# --- the same in float64 ---------------------------------------------------------------


def _interp(curve, t, outside_zero):
    if outside_zero and not curve[0][0] <= t <= curve[-1][0]:
        return 0.0
    return float(np.interp(t, [p[0] for p in curve], [p[1] for p in curve]))


def _where(c, a, b):
    return torch.where(c, a, torch.as_tensor(b, dtype=torch.float64, device="cuda"))


def _pad(t, axis, before, after):
    """t with zero slices added at both ends of one axis."""
    shape = list(t.shape)
    parts = []
    for n in (before, after):
        shape[axis] = n
        parts.append(torch.zeros(shape, dtype=t.dtype, device=t.device))
    return torch.cat([parts[0], t, parts[1]], dim=axis)


def _pair(t, axis):
    """The two cells of every interior face along an axis."""
    n = t.shape[axis]
    return t.narrow(axis, 0, n - 1), t.narrow(axis, 1, n - 1)


def _capacity(q, h, radius, n, d50):
    ok = (h >= H_DRY) & (q != 0)
    hs, rs = _where(ok, h, 1.0), _where(ok, radius, 1.0)
    theta = G * n * n * q * q / (hs * hs * rs ** (1.0 / 3.0)) / (1.65 * G * d50)
    qs = 8.0 * torch.clamp(theta - 0.047, min=0.0) ** 1.5 * math.sqrt(1.65 * G * d50**3)
    return _where(ok, torch.sign(q) * qs, 0.0)


def _manning(q, hf, slope, n, dt):
    wet = hf >= H_DRY
    hs = _where(wet, hf, 1.0)
    return _where(wet, (q - G * hs * dt * slope) / (1.0 + G * dt * n * n * q.abs() / hs ** (7.0 / 3.0)), 0.0)


class _LiExact:
    def __init__(self, c, d):
        self.c, self.dx = c, c["dx"]
        self.h, self.z = d["depth"].double(), d["bed"].double()
        n = d["manning"]
        self.n = n.double() if isinstance(n, torch.Tensor) else torch.full_like(self.h, float(np.float32(n)))
        ny, nx = self.h.shape
        zeros = lambda a, b: torch.zeros(a, b, dtype=torch.float64, device="cuda")  # noqa: E731
        self.q = [zeros(ny, nx + 1), zeros(ny + 1, nx)]
        self.qs = [zeros(ny, nx + 1), zeros(ny + 1, nx)] if c["sediment"] else None
        self.rain = d["rain_field"].double() if "rain_field" in d else (RAIN if c["rain"] == "uniform" else 0.0)
        self.infil = d["infil"].double() if "infil" in d else None
        self.open = {e for e, k in d.get("boundaries", {}).items() if k == "open"}
        self.inflows = d.get("inflows", []) if c["inflows"] else []
        self.t, self.ch = 0.0, None
        if c["channels"]:
            self.w, self.d = d["chan_w"].double(), d["chan_d"].double()
            self.cn = float(np.float32(0.03))
            self.ch = [zeros(ny, nx + 1), zeros(ny + 1, nx)]
            self.fp = [zeros(ny, nx + 1), zeros(ny + 1, nx)]

    def _curve(self, deep, over):
        """The storage curve: `deep` of a full-width depth below the banks, `over` above."""
        has = (self.w > 0) & (self.d > 0)
        bank = self.w * self.d / self.dx
        low = self.h * self.dx / _where(has, self.w, 1.0)
        return has, _where(self.h <= bank, deep + low, 0.0) + _where(self.h > bank, over + (self.h - bank), 0.0)

    def step(self):
        dx = self.dx
        eta, col = self.h + self.z, self.h
        if self.ch is not None:
            has, e = self._curve(self.z - self.d, self.z)
            eta = torch.where(has, e, eta)
            col = torch.where(has, self._curve(torch.zeros_like(self.h), self.d)[1], col)
        hm = float(col.max())
        dt = DT_MAX if hm <= H_DRY else min(ALPHA["local_inertial"] * dx / math.sqrt(G * hm), DT_MAX)
        h = self.h.clone()
        for (i, j), hydro in self.inflows:  # before the step; the wave speed above has not seen it
            h[i, j] += _interp(hydro, self.t + 0.5 * dt, True) * dt / (dx * dx)
        if self.inflows:
            self.h = h
            eta = h + self.z
            if self.ch is not None:
                has, e = self._curve(self.z - self.d, self.z)
                eta = torch.where(has, e, eta)
        face, parts = [], []
        for ax in (1, 0):
            k = 1 - ax
            (el, er), (zl, zr), (nl, nr) = _pair(eta, ax), _pair(self.z, ax), _pair(self.n, ax)
            top, bank, nf, slope = torch.maximum(el, er), torch.maximum(zl, zr), 0.5 * (nl + nr), (er - el) / dx
            inner = lambda t, ax=ax: t.narrow(ax, 1, t.shape[ax] - 2)  # noqa: E731
            if self.ch is None:
                q = _manning(inner(self.q[k]), top - bank, slope, nf, dt)
                parts.append((top, bank, nf))
            else:
                (wl, wr), (dl, dr) = _pair(self.w, ax), _pair(self.d, ax)
                wf, zc = torch.minimum(wl, wr), torch.maximum(zl - dl, zr - dr)
                qf = _manning(inner(self.fp[k]), top - bank, slope, nf, dt)
                hc = torch.minimum(top, bank) - zc
                on = (wf > 0) & (hc >= H_DRY)
                hs = _where(on, hc, 1.0)
                rad = _where(on, wf * hs / (wf + 2.0 * hs), 1.0)
                q0 = inner(self.ch[k])
                qc = (q0 - G * hs * dt * slope) / (1.0 + G * dt * self.cn**2 * q0.abs() / (hs * rad ** (4.0 / 3.0)))
                qc = _where(on, qc, 0.0)
                fr = wf / dx
                q = qf * (1.0 - fr) + qc * fr
                self.ch[k], self.fp[k] = _pad(qc, ax, 1, 1), _pad(qf, ax, 1, 1)
                parts.append((top, bank, nf, zc, wf))
            face.append(_pad(q, ax, 1, 1))
        qx, qy = face
        out = (torch.clamp(-qx[:, :-1], min=0) + torch.clamp(qx[:, 1:], min=0)
               + torch.clamp(-qy[:-1], min=0) + torch.clamp(qy[1:], min=0)) * (dt / dx)  # fmt: skip
        beta = _where(out > 0, torch.clamp(self.h / _where(out > 0, out, 1.0), 0.0, 1.0), 1.0)
        for ax in (1, 0):
            k = 1 - ax
            bl, br = _pair(beta, ax)
            q = face[k]
            inner = q.narrow(ax, 1, q.shape[ax] - 2)
            scale = _pad(torch.where(inner > 0, bl, torch.where(inner < 0, br, torch.ones_like(bl))), ax, 1, 1)
            face[k] = q * scale
            if self.ch is not None:
                self.ch[k], self.fp[k] = self.ch[k] * scale, self.fp[k] * scale
            if self.qs is not None:
                mid = lambda t, ax=ax: t.narrow(ax, 1, t.shape[ax] - 2)  # noqa: E731
                d50 = float(np.float32(0.002))
                top, bank, nf = parts[k][:3]
                hf = top - bank
                if self.ch is None:
                    cap = _capacity(mid(face[k]), hf, hf, nf, d50)
                else:
                    zc, wf = parts[k][3:]
                    hc = torch.minimum(top, bank) - zc
                    on = (wf > 0) & (hc >= H_DRY)
                    rad = _where(on, wf * hc / _where(on, wf + 2.0 * hc, 1.0), 1.0)
                    cch = _where(on, _capacity(mid(self.ch[k]), hc, rad, self.cn, d50), 0.0)
                    fr = wf / dx
                    cap = _capacity(mid(self.fp[k]), hf, hf, nf, d50) * (1.0 - fr) + cch * fr
                self.qs[k] = self.qs[k] + _pad(cap, ax, 1, 1) * dt
        qx, qy = self.q = face
        h = self.h + (qx[:, :-1] - qx[:, 1:] + qy[:-1] - qy[1:]) * (dt / dx) + self.rain * dt
        if self.infil is not None:
            h = h - torch.clamp(torch.minimum(self.infil * dt, h), min=0.0)
        ny, nx = h.shape
        for e, sl, q in (("west", (slice(None), 0), -qx[:, 1]), ("east", (slice(None), nx - 1), qx[:, nx - 1]),
                         ("north", (0,), -qy[1]), ("south", (ny - 1,), qy[ny - 1])):  # fmt: skip
            if e in self.open:
                h[sl] = h[sl] - torch.clamp(torch.minimum(torch.clamp(q, min=0.0) * (dt / dx), h[sl]), min=0.0)
        self.h = h
        self.t += dt

    def fields(self):
        out = {"h": self.h, "qx": self.q[0], "qy": self.q[1]}
        if self.ch is not None:
            out.update(qx_ch=self.ch[0], qx_fp=self.fp[0], qy_ch=self.ch[1], qy_fp=self.fp[1])
        if self.qs is not None:
            out.update(qs_int_x=self.qs[0], qs_int_y=self.qs[1])
        return out


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _hllc(hl, ul, vl, hr, ur, vr):
    """The HLLC flux (mass, normal and transverse momentum) with dry-bed wave speeds."""
    cl, cr = torch.sqrt(G * torch.clamp(hl, min=0)), torch.sqrt(G * torch.clamp(hr, min=0))
    dl, dr = hl <= H_DRY, hr <= H_DRY
    cs = (0.5 * (cl + cr) + 0.25 * (ul - ur)).abs()
    us = 0.5 * (ul + ur) + cl - cr
    sl = torch.where(dl, ur - 2 * cr, torch.where(dr, ul - cl, torch.minimum(ul - cl, us - cs)))
    sr = torch.where(dl, ur + cr, torch.where(dr, ul + 2 * cl, torch.maximum(ur + cr, us + cs)))
    gap = _where((sr - sl) != 0, sr - sl, 1.0)
    fl = (hl * ul, hl * ul * ul + 0.5 * G * hl * hl)
    fr = (hr * ur, hr * ur * ur + 0.5 * G * hr * hr)
    jump = (hr - hl, hr * ur - hl * ul)
    f = [torch.where(sl >= 0, a, torch.where(sr <= 0, b, (sr * a - sl * b + sl * sr * j) / gap))
         for a, b, j in zip(fl, fr, jump, strict=True)]  # fmt: skip
    den = hr * (ur - sr) - hl * (ul - sl)
    big = den.abs() > 1e-12
    star = torch.where(big, (sl * hr * (ur - sr) - sr * hl * (ul - sl)) / _where(big, den, 1.0), 0.5 * (ul + ur))
    none = dl & dr
    f = [_where(~none, x, 0.0) for x in f]
    return f[0], f[1], f[0] * torch.where(star >= 0, vl, vr)


class _HllcExact:
    def __init__(self, c, d):
        self.c, self.dx, self.d = c, c["dx"], d
        self.z = d["bed"].double()
        h = d["depth"]
        v = d.get("velocity")
        self.u = [h.double()] + [(h * v[k]).double() if v is not None else torch.zeros_like(self.z) for k in (0, 1)]
        n = d["manning"]
        self.n = n.double() if isinstance(n, torch.Tensor) else float(np.float32(n))
        self.rain = d["rain_field"].double() if "rain_field" in d else (RAIN if c["rain"] == "uniform" else 0.0)
        self.infil = d["infil"].double() if "infil" in d else None
        self.kind = {e: d.get("boundaries", {}).get(e, "closed") for e in EDGES}
        self.t = 0.0

    def _direction(self, h, un, ut, axis, stages):
        """Along one axis (columns for x): the face fluxes and the cells' bed source."""
        if axis == 0:
            h, un, ut, z = h.T, un.T, ut.T, self.z.T
        else:
            z = self.z
        ends = ("west", "east") if axis == 1 else ("north", "south")
        ext = lambda t: torch.cat([t[:, :1], t[:, :1], t, t[:, -1:], t[:, -1:]], dim=1)  # noqa: E731
        hp, zp, np_, tp = ext(h), ext(z), ext(un), ext(ut)
        e = hp + zp
        dry = (hp[:, 1:-1] <= H_DRY) | (hp[:, :-2] <= H_DRY) | (hp[:, 2:] <= H_DRY)
        fac = (~dry).double()
        slope = lambda t: fac * _minmod(t[:, 1:-1] - t[:, :-2], t[:, 2:] - t[:, 1:-1])  # noqa: E731
        vals = {}
        for key, t in (("e", e), ("z", zp), ("n", np_), ("t", tp)):
            s, m = slope(t), t[:, 1:-1]
            vals[key] = (m + 0.5 * s, m - 0.5 * s, s)
        # cells -1 .. n: the left cell of face j is cell j - 1, the right one cell j
        L = {k: v[0][:, :-1] for k, v in vals.items()}
        R = {k: v[1][:, 1:] for k, v in vals.items()}
        h_l, h_r = torch.clamp(L["e"] - L["z"], min=0), torch.clamp(R["e"] - R["z"], min=0)
        zs = torch.maximum(L["z"], R["z"])
        hls, hrs = torch.clamp(L["e"] - zs, min=0), torch.clamp(R["e"] - zs, min=0)
        f0, f1, f2 = _hllc(hls, L["n"], L["t"], hrs, R["n"], R["t"])
        fl, fr = f1 + 0.5 * G * (h_l**2 - hls**2), f1 + 0.5 * G * (h_r**2 - hrs**2)
        for j, edge, low in ((0, ends[0], True), (-1, ends[1], False)):
            if self.kind[edge] == "open":
                continue
            eh, en, et, ez = h[:, j], un[:, j], ut[:, j], z[:, j]
            if self.kind[edge] == "closed":
                gh, gn = eh, -en
            else:
                gh, gn = torch.clamp(stages[edge] - ez, min=0), en
            a = _hllc(gh, gn, et, eh, en, et) if low else _hllc(eh, en, et, gh, gn, et)
            f0[:, j], f2[:, j] = a[0], a[2]
            (fr if low else fl)[:, j] = a[1]
        src = -0.5 * G * (h_l[:, 1:] + h_r[:, :-1]) * vals["z"][2][:, 1:-1]
        res = (f0, fl, fr, f2, src)
        return tuple(t.T for t in res) if axis == 0 else res

    def _rates(self, u, dt, stages):
        h, hu, hv = u
        wet = h > H_DRY
        hs = _where(wet, h, 1.0)
        vx, vy = _where(wet, hu / hs, 0.0), _where(wet, hv / hs, 0.0)
        mx, xl, xr, xt, sx = self._direction(h, vx, vy, 1, stages)
        my, yl, yr, yt, sy = self._direction(h, vy, vx, 0, stages)
        out = (torch.clamp(-mx[:, :-1], min=0) + torch.clamp(mx[:, 1:], min=0)
               + torch.clamp(-my[:-1], min=0) + torch.clamp(my[1:], min=0)) * (dt / self.dx)  # fmt: skip
        beta = _where(out > 0, torch.clamp(h / _where(out > 0, out, 1.0), 0.0, 1.0), 1.0)
        one = torch.ones_like(beta)
        bx = torch.cat([one[:, :1], beta, one[:, :1]], dim=1)
        by = torch.cat([one[:1], beta, one[:1]], dim=0)
        mx = mx * torch.where(mx > 0, bx[:, :-1], bx[:, 1:])
        my = my * torch.where(my > 0, by[:-1], by[1:])
        dh = -((mx[:, 1:] - mx[:, :-1]) + (my[1:] - my[:-1])) / self.dx
        dhu = (-((xl[:, 1:] - xr[:, :-1]) + (yt[1:] - yt[:-1])) + sx) / self.dx
        dhv = (-((yl[1:] - yr[:-1]) + (xt[:, 1:] - xt[:, :-1])) + sy) / self.dx
        return dh, dhu, dhv

    def step(self):
        h, hu, hv = self.u
        wet = h > H_DRY
        hs = _where(wet, h, 1.0)
        speed = _where(wet, torch.maximum(hu.abs(), hv.abs()) / hs, 0.0) + torch.sqrt(G * torch.clamp(h, min=0))
        smax = float(speed.max())
        dt = DT_MAX if smax <= 0 else min(ALPHA["hllc_fv"] * self.dx / smax, DT_MAX)
        stages = {e: _interp(cv, self.t + 0.5 * dt, False) for e, cv in (self.d.get("stage") or {}).items()}
        r = self._rates(self.u, dt, stages)
        h1 = torch.clamp(h + dt * r[0], min=0)
        u1 = [h1] + [_where(h1 > H_DRY, a + dt * b, 0.0) for a, b in zip(self.u[1:], r[1:], strict=True)]
        r = self._rates(u1, dt, stages)
        hn = torch.clamp(0.5 * (h + h1 + dt * r[0]), min=0)
        w = hn > H_DRY
        mu, mv = (_where(w, 0.5 * (a + b + dt * k), 0.0) for a, b, k in zip(self.u[1:], u1[1:], r[1:], strict=True))
        den = 1.0 + G * dt * self.n * self.n * torch.sqrt(mu * mu + mv * mv) / _where(w, hn, 1.0) ** (7.0 / 3.0)
        hn = hn + self.rain * dt
        if self.infil is not None:
            hn = hn - torch.clamp(torch.minimum(self.infil * dt, hn), min=0.0)
        self.u = [hn, mu / den, mv / den]
        self.t += dt

    def fields(self):
        return {"h": self.u[0], "hu": self.u[1], "hv": self.u[2]}


def exact(case: dict, seed: int):
    def one(c, s):
        m = (_HllcExact if c["scheme"] == "hllc_fv" else _LiExact)(c, _inputs(c, s))
        for _ in range(c["steps"]):
            m.step()
        return m.fields()

    if case["api"] == "ensemble":
        return [one(m, seed * 1000 + k) for k, m in enumerate(_members(case))]
    return one(case, seed)
