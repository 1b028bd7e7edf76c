"""An implicit step whose block lists find no device memory (GPU).

The lists are an optimisation (64 bytes a tet): where they cannot be allocated the rows are
assembled one thread each, which needs none and gives the same bits for rows of up to 16
blocks.  The device's free memory is taken down to pieces too small for the lists before the
step that would build them.
"""
import ctypes as C

import numpy as np
import pytest

from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402


class TakenMemory:
    """Holds the free device memory in allocations down to a megabyte."""

    def __enter__(self):
        self.lib, self.held = C.CDLL("libcuda.so.1"), []
        size = 1 << 36
        while size >= 1 << 20:
            p = C.c_uint64()
            if self.lib.cuMemAlloc_v2(C.byref(p), C.c_size_t(size)) == 0:
                self.held.append(p)
            else:
                size >>= 1
        return self

    def __exit__(self, *_):
        for p in self.held:
            self.lib.cuMemFree_v2(p)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_the_step_runs_with_one_thread_rows(precision, monkeypatch):
    scene = meshes.config2()  # lists of 6 MB
    worlds = [SimWorld(scene, precision=precision) for _ in range(2)]
    monkeypatch.setenv("PK_ROW_KERNEL", "thread")
    for w in worlds:  # everything but the lists is allocated
        w.step()
        w.synchronize()
    worlds[0].step()
    monkeypatch.delenv("PK_ROW_KERNEL")
    with TakenMemory() as taken:
        assert taken.held
        worlds[1].step()
        worlds[1].synchronize()
    flags = worlds[1].cg_stats()["flags"]
    assert flags & L.FLAG_INTEGRATED, hex(flags)
    for a, b in zip(worlds[0].state(f64=True), worlds[1].state(f64=True)):
        np.testing.assert_array_equal(a, b)
    worlds[1].step()  # and the next one, with room again
    assert worlds[1].cg_stats()["flags"] & L.FLAG_INTEGRATED
