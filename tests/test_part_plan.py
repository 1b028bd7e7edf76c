"""Layout of the coupled part-resident PCG kernel, checked on the CPU (no GPU needed).

``pk_part_plan_selfcheck`` builds the full symmetric rows in the FP32 or the FP64 stream form,
checks every condition the kernel checks before it uses a part or a tile, that each halo row is
sent once, by its owner, to its place in the reader's window, and each block placed once (its
transpose once), and evaluates y = A x from the rows sent.  The product must equal the
symmetric upper-BSR product (SparseBlockMatrix::Multiply, src/Math/SparseBlockMatrix.cpp:209-268).
Sizes: one row; fewer rows than a tile, one tile and one row more in either form; parts on every
SM; the most rows of a block (3,840) and one more; rows longer than a pass of their lanes, the
longest a tile holds and one block more.
"""
import ctypes as C

import numpy as np
import pytest

from physik_b200 import _lib as L
from physik_b200 import meshes

from tests.test_ring_tiling import sym_upper_spmv
from tests.test_slab_plan import _pattern_and_coords

PRECISIONS = {"mixed": 1, "fp64": 2}


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def run(rs, col, coords, parts, precision, seed=0):
    n = len(rs) - 1
    rng = np.random.default_rng(seed)
    vals, x = rng.standard_normal(9 * len(col)), rng.standard_normal((n, 3))
    y, info = np.full((n, 3), np.nan), np.zeros(5, np.int32)
    coords = np.ascontiguousarray(coords, np.float64)
    rc = L.PK.pk_part_plan_selfcheck(n, _ptr(rs), _ptr(col), _ptr(vals), _ptr(x), _ptr(coords), parts,
                                     PRECISIONS[precision], _ptr(y), _ptr(info))
    if rc == 0:
        np.testing.assert_allclose(y, sym_upper_spmv(rs, col, vals, x), rtol=1e-12, atol=1e-10)
    return rc, info


def band(n, width):
    rows = [np.arange(r, min(n, r + width)) for r in range(n)]
    rs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    coords = np.zeros((n, 3))
    coords[:, 0] = np.arange(n)
    return rs, np.concatenate(rows).astype(np.int32), coords


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("parts", [1, 2, 7, 148])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 97, 500, 3840])
def test_banded_rows(n, parts, precision):
    rc, info = run(*band(n, 6), parts, precision, seed=n)
    assert rc == 0, L.last_error()
    assert info[0] == min(parts, n)
    assert (info[4] == 0) == (info[0] == 1)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_more_rows_than_a_block_holds_are_refused(precision):
    assert run(*band(3841, 2), 1, precision)[0] == L.PK_ERR_UNSUPPORTED
    assert run(*band(3841, 2), 2, precision)[0] == 0


@pytest.mark.parametrize("precision,cap", [("mixed", 512), ("fp64", 256)])
def test_rows_of_many_blocks(precision, cap):
    for n in (16, 17, 33, cap, cap + 1):  # row 0 coupled to all others
        rs = np.concatenate([[0], n + np.arange(n)]).astype(np.int32)
        col = np.concatenate([np.arange(n), np.arange(1, n)]).astype(np.int32)
        coords = np.random.default_rng(n).random((n, 3))
        for parts in (1, 3):
            rc, _ = run(rs, col, coords, parts, precision)
            assert rc == (0 if n <= cap else L.PK_ERR_UNSUPPORTED), (n, parts, L.last_error())


@pytest.mark.parametrize("precision", PRECISIONS)
def test_workload_bodies(precision):
    for scene, parts in ((meshes.config1(), 11), (meshes.config5(), 41), (meshes.config2(), 148),
                         (meshes.small_box(7, 3, 5), 1)):
        rs, col, coords = _pattern_and_coords(scene)
        rc, info = run(rs, col, coords, parts, precision)
        assert rc == 0, L.last_error()
        assert info[0] == parts


@pytest.mark.parametrize("precision", PRECISIONS)
def test_block128_on_all_sms(precision):
    rs, col, coords = _pattern_and_coords(meshes.config4())
    rc, info = run(rs, col, coords, 148, precision)
    assert rc == 0, L.last_error()
    assert info[1] <= 6144
