"""The bounded waits for tagged packets (resident and part-resident kernels), made to run out.

As in test_gpu_waits.py: a member of the exchange that was never launched, and a part that
sends none of its rows, cost a timeout status; the kernel leaves through its normal exit, and
the next launch on the same context is clean.
"""
import ctypes as C

import numpy as np
import pytest

from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

TIMEOUT, ENOUGH, FEW = -6, 1 << 22, 1 << 12
ROWS = 700


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def exchange(blocks, missing, limit):
    out = np.full((blocks, 4), -1.0)
    return L.PK.pk_tag_wait_selftest(0, blocks, missing, limit, _ptr(out)), out


def solve(kernel, lost, limit):
    x, iterations = np.full((ROWS, 3), np.nan), C.c_int(-1)
    rc = L.PK.pk_pcg_wait_selftest(0, kernel, lost, limit, _ptr(x), C.byref(iterations))
    return rc, x, iterations.value


@pytest.mark.parametrize("blocks", [2, 9, 33, 64])
def test_a_complete_group_exchanges(blocks):
    rc, out = exchange(blocks, 0, 1 << 16)
    assert rc == 0
    assert np.all(out[:, 0] == 1.0) and np.all(out[:, 3] == 0.0)
    assert np.all(out[:, 1] == blocks * (blocks + 1) / 2) and np.all(out[:, 2] == blocks)


@pytest.mark.parametrize("blocks,missing", [(2, 1), (16, 5), (64, 64)])
def test_a_missing_member_times_out(blocks, missing):
    rc, out = exchange(blocks, missing, FEW)
    assert rc == TIMEOUT
    assert np.all(out[:, 0] == 0.0) and np.all(out[:, 3] == 0.0)


@pytest.mark.parametrize("kernel", [0, 1, 2], ids=["resident", "cluster", "part"])
def test_rows_that_nobody_sends_time_out_and_the_next_solve_is_clean(kernel):
    rc, x, iterations = solve(kernel, 1, FEW)
    assert rc == TIMEOUT
    rc, x, iterations = solve(kernel, 0, ENOUGH)
    assert rc == 0 and 5 < iterations < 100
    a = 20.0 * x
    for k in range(1, 6):
        a[k:] -= x[:-k]
        a[:-k] -= x[k:]
    b = np.sin(3.0 * np.arange(ROWS)[:, None] + np.arange(3))
    assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
    w = SimWorld(meshes.small_box(3, 2, 2), precision="mixed")
    w.step()
    flags = w.cg_stats()["flags"]
    assert flags & L.FLAG_INTEGRATED and not flags & L.FLAG_BARRIER_TIMEOUT


def test_bad_arguments_are_refused_without_a_launch():
    out = np.zeros((4, 4))
    assert L.PK.pk_tag_wait_selftest(0, 1, 0, 100, _ptr(out)) == -3
    assert L.PK.pk_tag_wait_selftest(0, 4, 0, 0, _ptr(out)) == -3
    assert L.PK.pk_pcg_wait_selftest(0, 3, 0, 100, _ptr(out), _ptr(out)) == -3
