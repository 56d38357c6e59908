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
