"""FP64 steps whose solver pattern changes between them (GPU).

Point connections join the pattern; dragged from node to node they give every step another one.
A layout for the resident or the part-resident kernel costs the host more than such a step, so
a joined pattern that replaces a solved one starts on the ring kernel and gets its layout when it
has lasted; so does the first of a scene set again when tets were cut away.  A world's first pattern
and the bodies' own get it at once, the latter kept while others wait.  The kernels differ in the order of sums
only: against a world that always steps on the ring kernel within the FP64 tolerances of
test_gpu_resident.py, and with and without a captured step bit for bit.
"""
import numpy as np
import pytest

from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

RING = "pcg_ring_kernel"


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def connect(w, free, k):
    nodes = [int(free[(17 * k + 101 * j) % len(free)]) for j in range(4)]
    w.add_point_connection(nodes, (0.25,) * 4, (0.125, 0.25, 0.125), 40.0, 0.5)


@pytest.mark.parametrize("resident,kernel", [("1", "pcg_res_kernel"), ("0", "pcg_part_kernel")])
@pytest.mark.parametrize("graph", [False, True])
def test_a_pattern_that_lasts_gets_its_layout(graph, resident, kernel, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", resident)
    scene = meshes.small_box(9, 8, 7)
    free = np.nonzero(~scene.bodies[0].pinned)[0]
    w = SimWorld(scene, precision="fp64")
    w.set_graph(graph)
    names = []
    for k in range(9):  # plain, plain; another pattern each; the same one; none again
        if 2 <= k < 5:
            connect(w, free, k)
        elif 5 <= k < 7:
            connect(w, free, 4)
        w.step()
        assert w.cg_stats()["flags"] & L.FLAG_INTEGRATED
        names.append(w.pcg_launched())
    assert names == [kernel, kernel, RING, RING, RING, kernel, kernel, kernel, kernel]


def test_the_bodies_own_layout_is_kept_while_others_wait(monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")  # (building the part kernel's layout is one launch more)
    scene = meshes.small_box(9, 8, 7)
    free = np.nonzero(~scene.bodies[0].pinned)[0]
    w, plain = SimWorld(scene, precision="fp64"), SimWorld(scene, precision="fp64")
    w.enable_timing(True)
    names, launches = [], []
    for k in range(6):
        before = w.timings()["launches"]
        if k % 2:
            connect(w, free, k)
        w.step()
        names.append(w.pcg_launched())
        launches.append(w.timings()["launches"] - before)
    assert names == ["pcg_part_kernel", RING] * 3
    assert launches[2] == launches[4] == launches[0] - 1  # the layout is not built again
    x, v = w.state(f64=True)
    plain.prepare(True)
    plain.set_state(x, v, f64=True)
    for u in (w, plain):
        u.step()
        assert u.pcg_launched() == "pcg_part_kernel"
    for p, q in zip(w.state(f64=True), plain.state(f64=True)):
        np.testing.assert_array_equal(p, q)


@pytest.mark.parametrize("graph", [False, True])
def test_a_scene_set_again_waits_for_its_layout(graph, monkeypatch):
    scene = meshes.small_box(9, 8, 7)
    tets, pinned = scene.bodies[0].tets, scene.bodies[0].pinned
    counts = np.bincount(tets.ravel())
    corners = [n for n in np.argsort(counts, kind="stable") if not pinned[n]][:2]

    def run(w):
        names = []
        for k in range(7):
            if k in (2, 3):  # a corner node leaves the solve with its tets
                for t in np.nonzero((tets == corners[k - 2]).any(1))[0]:
                    w.X.PHYSIK_SetTetActive(w.h, w.components[0], int(t), 0)
            w.step()
            assert w.cg_stats()["flags"] & L.FLAG_INTEGRATED
            names.append(w.pcg_launched())
        return names, w.state(f64=True)

    w = SimWorld(scene, precision="fp64")
    w.set_graph(graph)
    names, (x, v) = run(w)
    assert names == ["pcg_res_kernel"] * 2 + [RING] * 2 + ["pcg_res_kernel"] * 3
    monkeypatch.setenv("PK_PCG_KERNEL", "ring")
    _, (x2, v2) = run(SimWorld(scene, precision="fp64"))
    assert rel(x, x2) <= 1e-12 and rel(v, v2) <= 1e-10


def test_the_wait_grows_with_the_rows():
    scene = meshes.small_box(33, 17, 16)  # 10,098 rows: two solves
    free = np.nonzero(~scene.bodies[0].pinned)[0]
    w = SimWorld(scene, precision="fp64")
    names = []
    for k in range(4):
        if k:
            connect(w, free, 1)
        w.step()
        names.append(w.pcg_launched())
    assert names == ["pcg_res_kernel", RING, RING, "pcg_res_kernel"]


def test_steps_equal_a_captured_world_and_follow_the_ring_kernel(monkeypatch):
    scene = meshes.small_box(9, 8, 7)
    free = np.nonzero(~scene.bodies[0].pinned)[0]
    worlds = [SimWorld(scene, precision="fp64") for _ in range(2)]
    worlds[1].set_graph(True)

    def run(w):
        for k in range(8):
            if k in (2, 3, 5, 6):
                connect(w, free, k // 2)
            w.step()
        return w.state(f64=True)

    (x0, v0), (x1, v1) = run(worlds[0]), run(worlds[1])
    np.testing.assert_array_equal(x0, x1)
    np.testing.assert_array_equal(v0, v1)
    monkeypatch.setenv("PK_PCG_KERNEL", "ring")
    x2, v2 = run(SimWorld(scene, precision="fp64"))
    assert rel(x0, x2) <= 1e-12 and rel(v0, v2) <= 1e-10


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_float_storage_does_not_wait(precision):
    scene = meshes.small_box(9, 8, 7)
    free = np.nonzero(~scene.bodies[0].pinned)[0]
    w = SimWorld(scene, precision=precision)
    for k in range(4):
        if k >= 2:
            connect(w, free, k)
        w.step()
        assert w.pcg_launched() == "pcg_res_kernel"
