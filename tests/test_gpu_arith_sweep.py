"""The step kernels' hand-written divisions, roots and powers over the ranges they state.

Exact build: reciprocal, square root, x / g and the 7/3 power equal the IEEE operations
(and rb_pow73f) on every float of their ranges, scalar and packed; the quotient on every
pair of exponents with random mantissas and with quotients next to a rounding midpoint.
The guarded forms built on them equal the general expression on operands of any bits.
Fast build: the approximate units' helpers stay within the bounds of their documentation.
"""

from __future__ import annotations

import ctypes
import importlib.util
import os
import subprocess

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKS = {
    "exact": ["reciprocal", "root", "power", "over_g", "quotient", "denominator", "manning", "slope", "riemann",
              "cell_values"],
    "fast": ["quotient", "root", "power"],
}


@pytest.fixture(scope="module")
def sweeps(tmp_path_factory):
    """The sweeps compiled with the product's own flags, one library per arithmetic."""
    spec = importlib.util.spec_from_file_location("rb_build", os.path.join(ROOT, "river-basin-sim_b200", "build.py"))
    rb = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(rb)
    out = tmp_path_factory.mktemp("arith")
    src = os.path.join(ROOT, "tests", "arith_sweep.cu")
    jobs = {}
    for mode, flags in (("exact", rb.EXACT), ("fast", rb.FAST)):
        cmd = [rb.nvcc(), *rb.ARCH, *rb.COMMON, *flags, "-cudart", "static", "-shared", "-I",
               os.path.join(ROOT, "include"), "-I", rb.CSRC, src, "-o", str(out / f"{mode}.so")]  # fmt: skip
        jobs[mode] = subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    for mode, job in jobs.items():
        said, _ = job.communicate()
        assert job.returncode == 0, f"{mode}: {said}"
    return {mode: ctypes.CDLL(str(out / f"{mode}.so")) for mode in jobs}


@pytest.mark.parametrize("mode, name", [(m, n) for m, names in CHECKS.items() for n in names])
def test_arithmetic_holds_over_its_range(sweeps, mode, name):
    tried, bad, first = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0), (ctypes.c_float * 2)()
    rc = getattr(sweeps[mode], f"sweep_{name}")(ctypes.byref(tried), ctypes.byref(bad), first)
    assert rc == 0 and tried.value > 0
    assert bad.value == 0, f"{bad.value} of {tried.value}, the first at ({first[0].hex()}, {first[1].hex()})"
