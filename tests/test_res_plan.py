"""Layout of the resident PCG kernel, checked on the CPU (no GPU needed).

``pk_res_plan_selfcheck`` cuts the rows into parts, deals each row's blocks to its lanes,
checks every condition the kernel checks before it uses a part, that each block is placed
once (and its transpose once) and that every halo row is sent by its owner inside the same
group, and evaluates y = A x as the kernel's lanes do.  The product must equal the
symmetric upper-BSR product (SparseBlockMatrix::Multiply,
src/Math/SparseBlockMatrix.cpp:209-268) computed with numpy.  Sizes: one row, one block's
worth of rows and one more, rows that fill a block's threads and one more, parts on every
lane count, in clusters and without, the largest that fits and one that does not.
"""
import ctypes as C

import numpy as np
import pytest

from physik_b200 import _lib as L
from physik_b200 import meshes

from tests.test_ring_tiling import sym_upper_spmv
from tests.test_slab_plan import _pattern_and_coords


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def run(rs, col, coords, seg=None, blocks=148, precision=1, seed=0):
    n = len(rs) - 1
    seg = np.array([0, n] if seg is None else seg, np.int32)
    rng = np.random.default_rng(seed)
    vals = rng.standard_normal(9 * len(col))
    x = rng.standard_normal((n, 3))
    y = np.full((n, 3), np.nan)
    info = np.zeros(6, np.int32)
    coords = np.ascontiguousarray(coords, np.float64)
    rc = L.PK.pk_res_plan_selfcheck(n, _ptr(rs), _ptr(col), _ptr(vals), _ptr(x), _ptr(coords), _ptr(seg),
                                    len(seg) - 1, blocks, precision, _ptr(y), _ptr(info))
    if rc == 0:
        np.testing.assert_allclose(y, sym_upper_spmv(rs, col, vals, x), rtol=1e-12, atol=1e-10)
    return rc, info


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("blocks", [1, 2, 7, 148, -2, -7, -148])  # negative: no clusters
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 96, 97, 128, 129, 255, 257])
def test_banded_rows(n, blocks, precision):
    """Every row couples to the next five, so that rows, parts and halos of odd sizes occur."""
    rows = [np.arange(r, min(n, r + 6)) for r in range(n)]
    rs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    coords = np.zeros((n, 3))
    coords[:, 0] = np.arange(n)
    rc, info = run(rs, col, coords, blocks=blocks, precision=precision, seed=n)
    if precision == 2 and n > 256 * abs(blocks):  # rows of 11 blocks on 288 threads exceed shared memory
        assert rc == L.PK_ERR_UNSUPPORTED
        return
    assert rc == 0, L.last_error()
    assert info[1] * info[2] <= info[5] and info[0] >= -(-n // info[1])
    assert info[4] == 0 or blocks > 0


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("blocks", [148, -148])
def test_workload_bodies(precision, blocks):
    for scene in (meshes.config1(), meshes.config5(), meshes.config2(), meshes.small_box(7, 3, 5)):
        rs, col, coords = _pattern_and_coords(scene)
        rc, info = run(rs, col, coords, blocks=blocks, precision=precision)
        assert rc == 0, L.last_error()
        assert info[2] in (1, 2, 4, 8)


def test_bodies_keep_their_own_groups_and_empty_bodies_have_none():
    scene = meshes.small_box(4, 3, 3)
    for i, shape in enumerate([(3, 5, 2), (9, 8, 7), (1, 1, 1)]):
        scene.bodies.append(meshes.small_box(*shape, seed=9 + i).bodies[0])
    rs, col, coords = _pattern_and_coords(scene)
    sizes = [int((~b.pinned).sum()) for b in scene.bodies]
    seg = np.concatenate([[0, 0], np.cumsum(sizes)])  # a body without rows first
    for blocks in (148, 16, -148):
        rc, info = run(rs, col, coords, seg=seg, blocks=blocks)
        assert rc == 0, L.last_error()
        assert info[0] >= 4
    rc, _ = run(rs, col, coords, seg=[0, sizes[0] - 1, len(rs) - 1])  # a cut through a body
    assert rc == L.PK_ERR_UNSUPPORTED


def test_a_matrix_larger_than_the_chip_is_refused():
    rs, col, coords = _pattern_and_coords(meshes.config4())
    assert run(rs, col, coords)[0] == L.PK_ERR_UNSUPPORTED
    rs, col, coords = _pattern_and_coords(meshes.config2())
    assert run(rs, col, coords, blocks=20)[0] == L.PK_ERR_UNSUPPORTED


def test_a_row_longer_than_the_registers_hold():
    """One row coupled to all others: more slots per lane than the registers hold."""
    n = 44
    rows = [np.arange(n)] + [np.array([r]) for r in range(1, n)]
    rs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    coords = np.random.default_rng(1).random((n, 3))
    for precision in (1, 2):
        for blocks in (1, 9, -9):
            rc, _ = run(rs, col, coords, blocks=blocks, precision=precision)
            assert rc == 0, L.last_error()
