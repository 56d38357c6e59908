"""Which step kernel a domain takes: the numbers that pin the 32 x 32 tiles, and what the
default chooses by size, by the names of the kernels that were launched."""

from __future__ import annotations

import re

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from cases import CASES, run_case  # noqa: E402

PINNED = {"local_inertial": 5, "hllc_fv": 9}
TILES = {"local_inertial": r"li_step_kernel<32, 32, 512,", "hllc_fv": r"hllc_stage_kernel<32, 32, 640,"}


@pytest.fixture(scope="module", autouse=True)
def _pow():
    oracle.set_pow_mode(1)
    yield
    oracle.set_pow_mode(0)


@pytest.fixture
def pin():
    """``pin(scheme)`` sets the 32 x 32 tiles for it; the variants in force come back after."""
    import ctypes

    from rbsim import _lib

    L = _lib.lib()
    li, hl, mode = ctypes.c_int32(), ctypes.c_int32(), ctypes.c_int32()
    _lib.check(L.rb_launch_config(ctypes.byref(li), ctypes.byref(hl), ctypes.byref(mode)))
    yield lambda scheme: _lib.check(
        (L.rb_hllc_set_kernel_variant if scheme == "hllc_fv" else L.rb_li_set_kernel_variant)(PINNED[scheme]))
    _lib.check(L.rb_li_set_kernel_variant(li.value))
    _lib.check(L.rb_hllc_set_kernel_variant(hl.value))


def step_kernels(run):
    """The names of the step kernels that ``run`` launches."""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    return {e.key for e in prof.key_averages() if re.search(r"li_step|hllc_stage|_stream_kernel", e.key)}


def one_step(scheme, ny, nx):
    import rbsim

    st = rbsim.State.from_bed(np.zeros((ny, nx), np.float32), 10.0, depth=0.5, manning=0.03)
    if scheme == "hllc_fv":
        st.arm_hllc_fields()
    sch = rbsim.get_scheme(scheme)
    return lambda: sch.step(st, dt=0.1, rain=0.0, rain_scale=1.0, t=0.0)


@pytest.mark.parametrize("shape", [(40, 70), (300, 420), (2308, 1300)], ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("arith_mode", ["exact", "fast"])
@pytest.mark.parametrize("scheme", sorted(PINNED))
def test_pinned_tiles_are_taken_at_any_size(scheme, arith_mode, shape, pin):
    from rbsim import arith

    pin(scheme)
    with arith.using(arith_mode):
        names = step_kernels(one_step(scheme, *shape))
    assert names and all(re.search(TILES[scheme], n) for n in names), names


@pytest.mark.parametrize("name", sorted(CASES))
def test_golden_cases_on_the_pinned_tiles_match_oracle_bitwise(name, pin):
    """The golden cases are small, so that by default they take the smallest tiles."""
    from gpu_api import GpuAPI
    from test_gpu_parity import _compare, _oracle_outputs

    case = CASES[name]()
    pin(case["scheme"])
    _compare(run_case(case, GpuAPI()), _oracle_outputs(case), name)


def _streaming_cases():
    from test_gpu_stream import HLLC_CASES, LI_CASES, NAN_CASES

    for name in sorted(LI_CASES):
        yield "li_" + name, LI_CASES[name], "exact"
    for name in sorted(HLLC_CASES):
        yield "hllc_" + name, HLLC_CASES[name], "exact"
    for name in sorted(NAN_CASES):
        yield "nan_" + name, NAN_CASES[name], "exact"
    for name in ("closed", "field_infil", "sediment"):
        yield "li_" + name, LI_CASES[name], "fast"
    for name in ("closed", "stage_plain_rain", "field_infil"):
        yield "hllc_" + name, HLLC_CASES[name], "fast"


@pytest.mark.parametrize("make, arith_mode", [pytest.param(m, a, id=f"{n}-{a}") for n, m, a in _streaming_cases()])
def test_streaming_tests_reach_the_streaming_kernels(make, arith_mode):
    """The sizes of test_gpu_stream.py stay above the limits of the dispatch."""
    from gpu_api import GpuAPI
    from rbsim import arith

    case = make()
    api, fast = GpuAPI(), arith_mode == "fast"
    with arith.using(arith_mode):
        st = api.make_state(case)
        names = step_kernels(lambda: api.step(st, 1e-3, case.get("rain", 0.0), 1.0, 0.0))
    want = "rb::fast::" if fast else "rb::"
    want += "hllc_stream_kernel<" if case["scheme"] == "hllc_fv" else "li_stream_kernel<"
    assert names and all(want in n for n in names), names


def _options(scheme, ny, nx):
    """Options whose code the tiles carry, by name."""
    from test_gpu_stream import MM_H, STAGES

    field = np.linspace(0.0, 80.0 * MM_H, ny * nx, dtype=np.float32).reshape(ny, nx)
    full = dict(rain_field=field, infil=np.full((ny, nx), 500.0 * MM_H, np.float32), boundaries={"east": "open"})
    if scheme == "hllc_fv":
        return {"field": full, "field_compensated": dict(full, compensated=True),
                "stage": dict(rain=50.0 * MM_H, stage_curves=STAGES,
                              boundaries={"east": "fixed_stage", "north": "fixed_stage", "west": "open"})}  # fmt: skip
    inf = np.full((ny, nx), np.inf, np.float32)
    bed = dict(d50=np.full((ny, nx), 0.002, np.float32), porosity=0.4, every=3, dz_lo=-inf, dz_hi=inf)
    return {"field": full, "field_compensated": dict(full, compensated=True),
            "bedload": dict(sediment=bed, compensated=True, rain=50.0 * MM_H, boundaries={"east": "open"}),
            "bedload_field": dict(full, sediment=bed)}  # fmt: skip


# the tile each size takes by default; ragged in both directions
BY_SIZE = [("local_inertial", 501, 397, TILES["local_inertial"], o)
           for o in ("field", "field_compensated", "bedload", "bedload_field")]
BY_SIZE += [("hllc_fv", 501, 433, TILES["hllc_fv"], o) for o in ("field", "field_compensated", "stage")]
BY_SIZE += [("hllc_fv", 301, 417, r"hllc_stage_kernel<32, 16, 640,", o) for o in ("field", "field_compensated")]


@pytest.mark.parametrize("scheme, ny, nx, kernel, option", BY_SIZE, ids=lambda v: str(v) if "<" not in str(v) else "")
def test_middle_sizes_take_their_tile_and_match_oracle_bitwise(scheme, ny, nx, kernel, option):
    from gpu_api import GpuAPI
    from test_gpu_parity import _compare, _oracle_outputs
    from test_gpu_stream import _hllc, _li

    case = (_hllc if scheme == "hllc_fv" else _li)(ny, nx, 21, **_options(scheme, ny, nx)[option])
    got = []
    names = step_kernels(lambda: got.append(run_case(case, GpuAPI())))
    assert names and all(re.search(kernel, n) for n in names), names
    _compare(got[0], _oracle_outputs(case), f"{scheme} {option}")
