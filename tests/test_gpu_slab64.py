"""The part-resident PCG kernel in FP64 (GPU): systems larger than the chip's memory.

The resident kernel is switched off, so that small boxes reach it: fewer rows than a tile,
tiles with remainders, many parts, one part of the most rows a block holds (3,840, ten records
a thread and 240 tiles), several parts of several records.  One teacher-forced step from the
same state against the FP64 oracle, with the FP64 tolerances of test_gpu_world.py: positions
1e-14, velocities 1e-12; the failure paths report what the other kernels report.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

CASES = [((1, 1, 1), 0), ((3, 1, 1), 0), ((5, 2, 2), 0), ((7, 3, 2), 1), ((13, 12, 11), 0), ((15, 15, 15), 1),
         ((21, 21, 20), 4), ((33, 17, 9), 2), ((41, 30, 29), 0)]


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("shape,blocks", CASES, ids=lambda c: str(c).replace(", ", "x"))
def test_sizes_follow_the_fp64_oracle(shape, blocks, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    scene = meshes.small_box(*shape)
    gpu = SimWorld(scene, precision="fp64")
    if blocks:
        gpu.prepare(True)
        assert gpu.set_pcg_grid(blocks) > 0
    ora = po.Oracle(scene, "f64", float_inputs=True)
    for _ in range(2):
        gpu.set_state(ora.x, ora.v, f64=True)
        gpu.step()
        ora.step()
        x, v = gpu.state(f64=True)
        st = gpu.cg_stats()
        assert st["flags"] & L.FLAG_INTEGRATED, hex(st["flags"])
        assert not blocks or gpu.pcg_kernel()[1] <= blocks
        assert rel(x, ora.x) <= 1e-14
        assert rel(v, ora.v) <= 1e-12
        assert abs(st["iterations"] - ora.last_stats()["iterations"]) <= 1


@pytest.mark.parametrize("iterations", [1, 2, 7])
def test_caps_repeats_and_graph_replay_match_the_ring_kernel(iterations, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    scene = meshes.config1()
    scene.max_iterations = iterations
    worlds = [SimWorld(scene, precision="fp64") for _ in range(2)]
    worlds[1].set_graph(True)
    for _ in range(4):
        for w in worlds:
            w.step()
    monkeypatch.setenv("PK_PCG_KERNEL", "ring")
    ring = SimWorld(scene, precision="fp64")
    for _ in range(4):
        ring.step()
    (x0, v0), (x1, v1), (x2, v2) = (w.state(f64=True) for w in worlds + [ring])
    np.testing.assert_array_equal(x0, x1)
    np.testing.assert_array_equal(v0, v1)
    a, b = worlds[0].cg_stats(), ring.cg_stats()
    assert a["iterations"] == b["iterations"] == iterations and a["flags"] == b["flags"]
    assert abs(a["residual"] - b["residual"]) <= 1e-8 * b["residual"]
    assert rel(x0, x2) <= 1e-12 and rel(v0, v2) <= 1e-10


def test_a_state_that_is_not_finite_is_not_integrated(monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    scene = meshes.small_box(4, 4, 4)
    flags = []
    for kernel in ("", "ring"):
        if kernel:
            monkeypatch.setenv("PK_PCG_KERNEL", kernel)
        w = SimWorld(scene, precision="fp64")
        w.step()
        x, v = w.state(f64=True)
        v = np.array(v)
        v[-1, 0] = np.inf
        w.set_state(x, v, f64=True)
        w.step()
        flags.append(w.cg_stats()["flags"])
        np.testing.assert_array_equal(w.state(f64=True)[0], x)
    assert flags[0] == flags[1] and not flags[0] & L.FLAG_INTEGRATED
