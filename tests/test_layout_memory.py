"""Layouts that find no host memory (CPU): a status, no exception through the C ABI.

A child process lowers its address-space limit to a little above what it uses, more at every
call, and asks the self-checks for layouts of a band of 120,000 rows: whatever allocation fails, the
call must return, with an error until the layout fits.
"""
import subprocess
import sys

import pytest

from physik_b200 import _lib as L

CHILD = r"""
import ctypes as C, os, resource, sys
# one thread: the C library ends a process whose new thread finds no memory for its local data
os.sched_setaffinity(0, {min(os.sched_getaffinity(0))})
sys.path.insert(0, sys.argv[1])
import numpy as np
from physik_b200 import _lib as L
kind = sys.argv[2]
n = 120000 if kind != "resident" else 60000
width = np.minimum(8, n - np.arange(n))
rs = np.concatenate([[0], np.cumsum(width)]).astype(np.int32)
col = (np.arange(rs[-1]) - np.repeat(rs[:-1], width) + np.repeat(np.arange(n), width)).astype(np.int32)
vals, x, y = np.ones(9 * len(col)), np.ones((n, 3)), np.zeros((n, 3))
coords, seg, info = np.zeros((n, 3)), np.array([0, n], np.int32), np.zeros(8, np.int32)
coords[:, 0] = np.arange(n)
p = lambda a: a.ctypes.data_as(C.c_void_p)
head = (n, p(rs), p(col), p(vals), p(x), p(coords))
calls = {
    "part64": lambda: L.PK.pk_part_plan_selfcheck(*head, 148, 2, p(y), p(info)),
    "part32": lambda: L.PK.pk_part_plan_selfcheck(*head, 148, 1, p(y), p(info)),
    "slab": lambda: L.PK.pk_slab_plan_selfcheck(*head, 148, 0, p(y), p(info)),
    "batched": lambda: L.PK.pk_slab_plan_batched_selfcheck(*head, p(seg), 1, 148, 0, p(y), p(info)),
    "resident": lambda: L.PK.pk_res_plan_selfcheck(*head, p(seg), 1, 148, 1, p(y), p(info)),
}
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
hard = resource.getrlimit(resource.RLIMIT_AS)[1]
results = []
for mb in list(range(1, 40, 3)) + [60, 90, 130, 180, 260]:
    resource.setrlimit(resource.RLIMIT_AS, (used + (mb << 20), hard))
    results.append(calls[kind]())
resource.setrlimit(resource.RLIMIT_AS, (hard, hard))
results.append(calls[kind]())
print(*results)
"""


@pytest.mark.parametrize("kind", ["part64", "part32", "slab", "batched", "resident"])
def test_a_call_without_memory_returns_an_error(kind):
    child = subprocess.run([sys.executable, "-c", CHILD, L.ROOT, kind], capture_output=True, text=True, timeout=300)
    assert child.returncode == 0, (child.returncode, child.stderr[-500:])
    results = [int(r) for r in child.stdout.split()]
    assert results[-1] == 0 and any(r < 0 for r in results)
    assert set(results) <= {0, L.PK_ERR_UNSUPPORTED}, results
