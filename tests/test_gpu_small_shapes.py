"""What small domains take: tiles chosen by the domain's size, and compute_dt's reduction in
one launch."""

from __future__ import annotations

import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle  # noqa: E402
from cases import run_case  # noqa: E402
from test_gpu_stream import ALL_OPEN, MM_H, _hllc, _li  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _pow():
    oracle.set_pow_mode(1)
    yield
    oracle.set_pow_mode(0)


# One cell, one 16 x 16 tile and its remainders; narrow and flat domains, whose 16 x 16 tiles
# outnumber the ledger's slots; either side of the LI limit (100 000 cells) and of the HLLC
# ones (75 000 and 200 000).
SHAPES = [(1, 1), (16, 16), (17, 33), (15, 47), (200, 3), (3, 200), (400, 250), (401, 250), (300, 250), (301, 250),
          (400, 500), (401, 500)]  # fmt: skip


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("scheme", ["li", "hllc"])
def test_tiles_by_size_match_oracle_bitwise(scheme, shape):
    from gpu_api import GpuAPI
    from test_gpu_parity import _compare, _oracle_outputs

    ny, nx = shape
    make = _li if scheme == "li" else _hllc
    case = make(ny, nx, 11, compensated=True, rain=50.0 * MM_H, boundaries=ALL_OPEN,
                infil=np.full((ny, nx), 2000.0 * MM_H, np.float32))  # fmt: skip
    _compare(run_case(case, GpuAPI()), _oracle_outputs(case), f"{scheme} {ny}x{nx}")


def _state(ny, nx, depth):
    import rbsim

    return rbsim.State.from_bed(np.zeros((ny, nx), np.float32), 10.0, depth=depth, manning=0.03)


# fewer cells than a block, a block's remainders, more than all blocks hold at once
@pytest.mark.parametrize("n", [1, 31, 1023, 1025, 1184 * 1024 * 2 + 1])
def test_dt_is_that_of_the_largest_depth_wherever_it_is(n):
    from rbsim.schemes import local_inertial as li

    for at in sorted({0, n // 2, n - 1}):
        depth = torch.full((1, n), 0.01)
        depth[0, at] = 1.5 + at / n
        want = 0.7 * 10.0 / float(np.sqrt(9.81 * float(depth.max())))
        got = li.compute_dt(_state(1, n, depth.numpy()), 0.7, dt_max=1e9)
        assert got == pytest.approx(want, rel=1e-15)


def test_dt_from_several_threads_and_streams():
    """A call holds a result word of its own: eight threads, on their own streams, read the dt
    of their own state every time."""
    from rbsim.schemes import local_inertial as li

    wrong = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            st = _state(64, 64, np.full((64, 64), 0.1 * (k + 1), np.float32))
            torch.cuda.current_stream().synchronize()
            want = 0.7 * 10.0 / float(np.sqrt(9.81 * float(np.float32(0.1 * (k + 1)))))
            wrong.extend(k for _ in range(50) if li.compute_dt(st, 0.7, dt_max=1e9) != pytest.approx(want, rel=1e-15))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
