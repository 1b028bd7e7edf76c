"""The coupled part-resident PCG kernel in FP32 storage (GPU), reached by small boxes with the
resident kernel switched off: fewer rows than a tile, tiles with remainders, many parts, one
part of the most rows (3,840), several parts of several records.  One teacher-forced step from
the same state against the FP64 oracle, with the FP32-storage tolerances of
test_gpu_resident.py (positions 3e-7, velocities 2e-4); repeats and graph replay bit for bit.
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


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("shape,blocks", CASES, ids=lambda c: str(c).replace(", ", "x"))
def test_sizes_follow_the_fp64_oracle(shape, blocks, precision, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    scene = meshes.small_box(*shape)
    gpu = SimWorld(scene, precision=precision)
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
        kernel, used = gpu.pcg_kernel()
        assert kernel == "slab" and (not blocks or used <= blocks)
        assert rel(x, ora.x) <= 3e-7
        assert rel(v, ora.v) <= 2e-4
        assert abs(st["iterations"] - ora.last_stats()["iterations"]) <= 1


@pytest.mark.parametrize("iterations", [1, 2, 7, 100])
def test_repeats_and_graph_replay_are_bit_identical(iterations, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    scene = meshes.config2()
    scene.max_iterations = iterations
    worlds = [SimWorld(scene, precision="mixed") for _ in range(3)]
    worlds[2].set_graph(True)
    for _ in range(4):
        for w in worlds:
            w.step()
    x, v = worlds[0].state(f64=True)
    assert worlds[0].cg_stats()["iterations"] <= iterations
    for w in worlds[1:]:
        np.testing.assert_array_equal(w.state(f64=True)[0], x)
        np.testing.assert_array_equal(w.state(f64=True)[1], v)
