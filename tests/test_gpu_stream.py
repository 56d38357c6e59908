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


def test_li_streaming_flags_a_non_finite_depth():
    import rbsim
    from rbsim import _lib

    st = rbsim.State.from_bed(np.zeros((1429, 1400), np.float32), 10.0, depth=1.0, manning=0.03)
    h = np.ones((1429, 1400), np.float32)
    h[700, 27] = np.nan
    st.h = h
    rbsim.get_scheme("local_inertial").step(st, 0.5)
    with pytest.raises(_lib.DeviceError):
        st.check_device_errors()
