"""The layout self-checks write as many values to `info` as the header promises (CPU)."""
import ctypes as C
import re

import numpy as np
import pytest

from physik_b200 import _lib as L

GUARD = -77777


def documented(function):
    """How many values the header's comment on the function lists after "info ... receives"."""
    text = open(L.HEADERS[0]).read()
    comment = text[:text.index(f"PKCUDA_API int {function}(")].rsplit("/*", 1)[1]
    return len(re.search(r"receives\s*\{([^}]*)\}", comment).group(1).split(","))


@pytest.mark.parametrize("function", ["pk_slab_plan_selfcheck", "pk_slab_plan_batched_selfcheck",
                                      "pk_res_plan_selfcheck"])
def test_info_has_the_documented_length(function):
    n = 40
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rs, col = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    vals, x, y, coords = np.ones(9 * n), np.ones((n, 3)), np.zeros((n, 3)), np.zeros((n, 3))
    info, seg = np.full(16, GUARD, np.int32), np.array([0, n], np.int32)
    more = {"pk_slab_plan_selfcheck": (3, 0), "pk_slab_plan_batched_selfcheck": (p(seg), 1, 4, 0),
            "pk_res_plan_selfcheck": (p(seg), 1, 4, 1)}[function]
    rc = getattr(L.PK, function)(n, p(rs), p(col), p(vals), p(x), p(coords), *more, p(y), p(info))
    assert rc == 0, L.last_error()
    assert int((info != GUARD).sum()) == documented(function)
    assert np.all(info[documented(function):] == GUARD)
