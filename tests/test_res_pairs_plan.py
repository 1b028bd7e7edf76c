"""The resident layout with two rows a thread and with slots in tensor memory: the host checks
the plan's conditions and multiplies through it (pk_res_plan_selfcheck), at the part sizes
around its limits (257 rows, the first with two rows a thread; 640, the most), for rows of one
block and of many."""
import ctypes as C

import numpy as np
import pytest

L = pytest.importorskip("physik_b200._lib")


def run(n, width, blocks, precision):
    rows = [np.arange(r, min(n, r + width)) for r in range(n)]
    rs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    rng = np.random.default_rng(n + width)
    vals, x = rng.standard_normal((len(col), 9)), rng.standard_normal((n, 3))
    coords = np.stack([np.arange(n), np.zeros(n), np.zeros(n)], axis=1).astype(np.float64)
    seg, y, info = np.array([0, n], np.int32), np.full((n, 3), np.nan), np.zeros(8, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rc = L.PK.pk_res_plan_selfcheck(n, p(rs), p(col), p(vals), p(x), p(coords), p(seg), 1, blocks, precision, p(y), p(info))
    want = np.zeros((n, 3))
    for r in range(n):
        for k in range(rs[r], rs[r + 1]):
            b = vals[k].reshape(3, 3).T  # column-major
            want[r] += b @ x[col[k]]
            if col[k] != r:
                want[col[k]] += b.T @ x[r]
    return rc, info, y, want


@pytest.mark.parametrize("per,width", [(257, 4), (300, 1), (320, 7), (321, 7), (500, 8), (600, 8), (640, 7)])
@pytest.mark.parametrize("blocks", [-1, -3])
def test_two_rows_a_thread(per, width, blocks):
    rc, info, y, want = run(per * -blocks, width, blocks, 1)
    assert rc == 0, L.last_error()
    assert info[1] == per and info[2] == 1 and info[5] >= per
    assert np.abs(y - want).max() <= 1e-11


@pytest.mark.parametrize("per", [240, 256])
def test_fp64_slots_in_tensor_memory(per):
    rc, info, y, want = run(3 * per, 8, -3, 2)
    assert rc == 0, L.last_error()
    assert info[1] == per and info[5] >= per
    assert np.abs(y - want).max() <= 1e-11


def test_more_rows_than_a_block_holds_are_refused():
    assert run(641, 2, -1, 1)[0] == L.PK_ERR_UNSUPPORTED
    assert run(600, 40, -1, 1)[0] == L.PK_ERR_UNSUPPORTED
