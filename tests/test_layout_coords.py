"""Layouts cut from coordinates that are not finite, on the CPU.

A state may hold NaN or infinite positions (the step then reports it and integrates nothing),
and the layouts' cuts sort by them.  A coordinate that is not finite counts as 0, so that the
layout, and with it every bit of its product, is the one that 0 in its place gives, or the
same refusal.
"""
import ctypes as C

import numpy as np
import pytest

from physik_b200 import _lib as L

BAD = [np.nan, np.inf, -np.inf]


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def band(n):
    rows = [np.arange(r, min(n, r + 6)) for r in range(n)]
    return (np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32),
            np.concatenate(rows).astype(np.int32))


def product(kind, n, coords):
    rs, col = band(n)
    rng = np.random.default_rng(n)
    vals, x = rng.standard_normal(9 * len(col)), rng.standard_normal((n, 3))
    y, info = np.full((n, 3), np.nan), np.zeros(8, np.int32)
    head = (n, _ptr(rs), _ptr(col), _ptr(vals), _ptr(x), _ptr(coords))
    if kind == "resident":
        rc = L.PK.pk_res_plan_selfcheck(*head, _ptr(np.array([0, n], np.int32)), 1, -23, 1, _ptr(y), _ptr(info))
    elif kind == "batched":
        rc = L.PK.pk_slab_plan_batched_selfcheck(*head, _ptr(np.array([0, n], np.int32)), 1, 8, 0, _ptr(y), _ptr(info))
    else:
        rc = L.PK.pk_slab_plan_selfcheck(*head, 7, 1 if kind == "symmetric" else 0, _ptr(y), _ptr(info))
    return rc, y, info


@pytest.mark.parametrize("bad", BAD, ids=str)
@pytest.mark.parametrize("kind", ["full", "symmetric", "batched", "resident"])
@pytest.mark.parametrize("n", [50, 400, 2500, 9000])
def test_a_coordinate_that_is_not_finite_counts_as_zero(kind, n, bad):
    rng = np.random.default_rng(n)
    coords = rng.uniform(-50, 50, (n, 3))
    coords[:, 0] = np.arange(n)
    at = rng.random((n, 3)) < 0.1
    zeros = np.where(at, 0.0, coords)
    rc0, y0, info0 = product(kind, n, zeros)
    rc1, y1, info1 = product(kind, n, np.where(at, bad, coords))
    assert rc0 == rc1 and (rc0 == 0 or n > 400), L.last_error()
    np.testing.assert_array_equal(info1, info0)
    np.testing.assert_array_equal(y1, y0)
