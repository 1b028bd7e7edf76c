"""An explicit step launches its two kernels and nothing else (GPU): the block lists that
implicit steps read and the solve's layout are not built for it, and are once an implicit step
follows."""
import pytest

from physik_b200 import meshes

pytestmark = pytest.mark.gpu

pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("graph", [False, True])
def test_an_explicit_step_is_two_launches(graph, precision, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")  # (the part kernel's FP64 layout is a launch)
    w = SimWorld(meshes.small_box(4, 3, 2), precision=precision, implicit=False)
    w.prepare(True)
    w.set_graph(graph)
    w.enable_timing(True)
    launches = []
    for _ in range(4):
        w.step()
        w.synchronize()
        launches.append(w.timings()["launches"])
    first = launches[0]
    assert [n - first for n in launches] == [0, 2, 4, 6] and first == 2, launches
    w.X.PHYSIK_SetSolverMode(w.h, 1)
    w.step()
    w.synchronize()
    assert w.timings()["launches"] >= launches[-1] + 4  # the lists, tets, rows and the solve
