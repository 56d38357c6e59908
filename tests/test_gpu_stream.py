"""The row-streaming step kernels at the sizes only they take (millions of cells) and at
the edges of their strips and chunks, against the oracle: bit for bit in the exact build,
to the solver tolerance in the fast one."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from cases import run_case  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _pow():
    if not torch.cuda.is_available():
        pytest.fail("the gpu tests need a CUDA device")
    oracle.set_pow_mode(1)
    yield
    oracle.set_pow_mode(0)


def _with_nan(a, cells):
    a = a.copy()
    for c in cells:
        a[c] = np.nan
    return a


def _li(ny, nx, seed, dx=10.0, **more):
    """Bumps with wet, drying and dry cells, uneven roughness, water already moving."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:ny, 0:nx].astype(np.float32)
    z = (1e-3 * x + 0.8 * np.sin(0.11 * x) * np.cos(0.07 * y) + 0.3 * np.sin(0.9 * y)).astype(np.float32)
    depth = np.maximum(rng.uniform(-0.2, 0.5, (ny, nx)), 0.0).astype(np.float32)
    depth[:, nx // 3 : nx // 2] = 0.0
    case = dict(scheme="local_inertial", bed=z, dx=dx, depth=depth, steps=6, alpha=0.7, dt_max=30.0,
                manning=rng.uniform(0.02, 0.06, (ny, nx)).astype(np.float32))  # fmt: skip
    case.update(more)
    return case


ALL_OPEN = {e: "open" for e in ("north", "south", "east", "west")}
MM_H = 1.0 / 3.6e6

# 1429 x 1400: a last strip with all 28 columns; 1001 x 2003: ragged in both, 15 of 28
# columns in the last strip, short last chunk; 72 x 28001: one column in the last strip.
LI_CASES = {
    "closed": lambda: _li(1429, 1400, 1),
    "rain_open": lambda: _li(1001, 2003, 2, compensated=True, rain=50.0 * MM_H, boundaries=ALL_OPEN),
    "plain_rain": lambda: _li(1429, 1400, 3, rain=50.0 * MM_H, boundaries={"west": "open"}),
    "field_infil": lambda: _li(1001, 2003, 4, compensated=True, boundaries=ALL_OPEN,
                               rain_field=np.full((1001, 2003), 40.0 * MM_H, np.float32),
                               infil=np.full((1001, 2003), 2000.0 * MM_H, np.float32)),
    "field_plain": lambda: _li(72, 28001, 5, rain_field=np.full((72, 28001), 40.0 * MM_H, np.float32)),
    "flat_wide": lambda: _li(72, 28001, 6, compensated=True, rain=50.0 * MM_H, boundaries=ALL_OPEN),
    "sediment": lambda: _li(1001, 2003, 7, boundaries={"east": "open"}, compensated=True, rain=50.0 * MM_H,
                            sediment=dict(d50=np.full((1001, 2003), 0.002, np.float32), porosity=0.4, every=3,
                                          dz_lo=np.full((1001, 2003), -np.inf, np.float32),
                                          dz_hi=np.full((1001, 2003), np.inf, np.float32))),
    # a cell size outside the range of the shared reciprocal: every face divides
    "huge_cells": lambda: _li(1429, 1400, 8, dx=4194304.0),
    # near-still water: discharges and surface differences down to the rounding of eta
    "still": lambda: _li(1429, 1400, 9, bed=np.zeros((1429, 1400), np.float32),
                         depth=(1.0 + 1e-7 * np.arange(1400, dtype=np.float32)[None, :]
                                * np.ones((1429, 1), np.float32)).astype(np.float32), manning=0.0),
}  # fmt: skip


@pytest.mark.parametrize("name", sorted(LI_CASES))
def test_li_streaming_matches_oracle_bitwise(name):
    from gpu_api import GpuAPI
    from test_gpu_parity import _compare, _oracle_outputs

    case = LI_CASES[name]()
    _compare(run_case(case, GpuAPI()), _oracle_outputs(case), name)


@pytest.mark.parametrize("name", ["closed", "field_infil", "sediment"])
def test_li_streaming_fast_within_tolerance(name):
    """The bound of test_gpu_fast_arith.py for random depths around the dry threshold."""
    from gpu_api import GpuAPI
    from rbsim import arith
    from test_gpu_fast_arith import _close, _fixed_dt

    case = LI_CASES[name]()
    with arith.using("fast"):
        got = run_case(dict(case), GpuAPI())
    _close(got, _fixed_dt(case, got), name, max_depth_m=1e-3, rel=2e-5)


def _hllc(ny, nx, seed, **more):
    """Moving water over bumps, some of them dry, with uneven roughness."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:ny, 0:nx].astype(np.float32)
    z = (0.6 + 0.9 * np.sin(0.05 * x) * np.cos(0.07 * y)).astype(np.float32)
    depth = np.maximum(1.0 + 0.2 * np.sin(0.3 * x + 0.2 * y) - z, 0.0).astype(np.float32)
    vel = rng.uniform(-1.0, 1.0, (2, ny, nx)).astype(np.float32)
    case = dict(scheme="hllc_fv", bed=z, dx=2.0, depth=depth, hu0=depth * vel[0], hv0=depth * vel[1], steps=4,
                alpha=0.45, dt_max=30.0, manning=rng.uniform(0.0, 0.05, (ny, nx)).astype(np.float32))  # fmt: skip
    case.update(more)
    return case


STAGES = {"east": [(0.0, 1.4), (1.0e4, 0.9)], "north": [(0.0, 0.8), (1.0e4, 1.3)]}

# 2308 x 1300: a last strip with all 26 columns; 1501 x 2003: one column in the last strip;
# 135 x 23000: a flat domain with a short last chunk.
HLLC_CASES = {
    "closed": lambda: _hllc(2308, 1300, 1),
    "open_rain": lambda: _hllc(1501, 2003, 2, compensated=True, rain=50.0 * MM_H, boundaries=ALL_OPEN),
    "stage_plain_rain": lambda: _hllc(135, 23000, 3, rain=50.0 * MM_H, stage_curves=STAGES,
                                      boundaries={"east": "fixed_stage", "north": "fixed_stage", "west": "open"}),
    "field_infil": lambda: _hllc(1501, 2003, 4, compensated=True, boundaries={"south": "open"},
                                 rain_field=np.full((1501, 2003), 40.0 * MM_H, np.float32),
                                 infil=np.full((1501, 2003), 2000.0 * MM_H, np.float32)),
    # still water with islands: zero velocities, zero contact speeds, rest at the shore
    "still": lambda: _hllc(2308, 1300, 5, hu0=np.zeros((2308, 1300), np.float32),
                           hv0=np.zeros((2308, 1300), np.float32)),
    # momenta down to the subnormals and depths up to 1e5: outside the quick divisions
    "odd_operands": lambda: _hllc(1501, 2003, 6, hu0=np.full((1501, 2003), 1e-39, np.float32),
                                  hv0=np.full((1501, 2003), -1e-25, np.float32), bed=np.zeros((1501, 2003), np.float32),
                                  depth=np.logspace(-6, 5, 2003, dtype=np.float32)[None, :].repeat(1501, 0)),
}  # fmt: skip


NAN_CASES = {
    # depths that are not numbers, inside a strip, at its edge and on the domain's edge
    "li": lambda: _li(1429, 1400, 10, steps=3, depth=_with_nan(
        np.full((1429, 1400), 0.3, np.float32), [(700, 700), (1000, 27), (1001, 28), (0, 5), (1428, 1399)])),
    # depths and momenta that are not numbers
    "hllc": lambda: _hllc(2308, 1300, 7, steps=2, hu0=_with_nan(np.ones((2308, 1300), np.float32), [(800, 800), (51, 26)]),
                         depth=_with_nan(np.ones((2308, 1300), np.float32), [(700, 700), (50, 25), (0, 4), (2307, 9)])),
}  # fmt: skip


@pytest.mark.parametrize("name", sorted(HLLC_CASES))
def test_hllc_streaming_matches_oracle_bitwise(name):
    from gpu_api import GpuAPI
    from test_gpu_parity import _compare, _oracle_outputs

    case = HLLC_CASES[name]()
    _compare(run_case(case, GpuAPI()), _oracle_outputs(case), name)


@pytest.mark.parametrize("name", ["closed", "stage_plain_rain", "field_infil"])
def test_hllc_streaming_fast_within_tolerance(name):
    from gpu_api import GpuAPI
    from rbsim import arith
    from test_gpu_fast_arith import _close, _fixed_dt

    case = HLLC_CASES[name]()
    with arith.using("fast"):
        got = run_case(dict(case), GpuAPI())
    _close(got, _fixed_dt(case, got), name, max_depth_m=1e-3, rel=2e-5)


@pytest.mark.parametrize("scheme", ["li", "hllc"])
def test_streaming_spreads_and_flags_nan_as_the_oracle_does(scheme, monkeypatch):
    """Depths and momenta that are not numbers reach the same cells as in the reference's
    expressions, and the step flags them."""
    import rbsim
    from gpu_api import GpuAPI
    from rbsim import _lib
    from test_gpu_parity import _compare, _oracle_outputs

    check, raised = rbsim.State.check_device_errors, []

    def note(st):
        try:
            check(st)
        except _lib.DeviceError as e:
            raised.append(str(e))

    monkeypatch.setattr(rbsim.State, "check_device_errors", note)
    case = NAN_CASES[scheme]()
    _compare(run_case(case, GpuAPI()), _oracle_outputs(case), scheme)
    assert raised
