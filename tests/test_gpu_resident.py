"""The resident PCG kernel (the matrix on chip for the whole solve) on the GPU.

It runs wherever the whole matrix fits the SMs' on-chip memory, in place of the streaming
kernels.  One teacher-forced step from the same state is compared with the FP64 oracle (the
reference's CPU solve in double) with the tolerances that the streaming kernels' tests use
(``test_gpu_slab.py``, ``test_gpu_world.py``): FP64 positions 1e-14 and velocities 1e-12,
FP32 storage positions 3e-7 and velocities 2e-4.  Sizes: one dynamic row of blocks, bodies
on one block of the launch (up to its row limit), on thread-block clusters of every size,
and on all SMs through global memory; bodies of their own in one batched launch, with more
clusters than are resident at once; against the streaming kernels on the same step.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

TOL = {"fp64": (1e-14, 1e-12), "mixed": (3e-7, 2e-4), "fp32": (3e-7, 2e-4)}


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


SHAPES = [(1, 1, 1), (4, 3, 2), (6, 4, 3), (7, 7, 6), (9, 9, 9), (13, 12, 11), (17, 16, 15), (33, 9, 8), (41, 21, 17)]


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_sizes_follow_the_fp64_oracle(shape, precision):
    scene = meshes.small_box(*shape)
    gpu = SimWorld(scene, precision=precision)
    ora = po.Oracle(scene, "f64", float_inputs=True)
    for _ in range(2):
        gpu.set_state(ora.x, ora.v, f64=True)
        gpu.step()
        ora.step()
        x, v = gpu.state(f64=True)
        st = gpu.cg_stats()
        assert st["flags"] & L.FLAG_INTEGRATED, hex(st["flags"])
        assert rel(x, ora.x) <= TOL[precision][0]
        assert rel(v, ora.v) <= TOL[precision][1]
        assert abs(st["iterations"] - ora.last_stats()["iterations"]) <= 1


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("iterations", [1, 2, 3, 7])
def test_iteration_caps_match_the_streaming_kernels(precision, iterations, monkeypatch):
    scene = meshes.config2()
    scene.max_iterations = iterations
    res = SimWorld(scene, precision=precision)
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    ref = SimWorld(scene, precision=precision)
    ref.step()
    monkeypatch.delenv("PK_PCG_RESIDENT")
    res.step()
    a, b = res.cg_stats(), ref.cg_stats()
    assert a["iterations"] == b["iterations"] == iterations and a["flags"] == b["flags"]
    assert abs(a["residual"] - b["residual"]) <= 1e-5 * b["residual"]
    (xa, va), (xb, vb) = res.state(f64=True), ref.state(f64=True)
    assert rel(xa, xb) <= TOL[precision][0] and rel(va, vb) <= TOL[precision][1]


@pytest.mark.parametrize("count,lo,hi", [(3, 1, 3), (40, 2, 8), (300, 1, 6)])
def test_batched_bodies_match_the_streaming_kernel(count, lo, hi, monkeypatch):
    rng = np.random.default_rng(count)
    scene = meshes.small_box(*(int(c) for c in rng.integers(lo, hi + 1, 3)))
    for i in range(count - 1):
        scene.bodies += meshes.small_box(*(int(c) for c in rng.integers(lo, hi + 1, 3)), seed=i).bodies
    for b in scene.bodies:
        b.initial_velocities = np.tile(rng.normal(0, 0.5, 3), (len(b.positions), 1)).astype(np.float32)
        b.initial_velocities[b.pinned] = 0.0
    worlds = []
    for resident in ("0", "1"):
        monkeypatch.setenv("PK_PCG_RESIDENT", resident)
        w = SimWorld(scene, precision="mixed")
        w.set_batched(True)
        w.step()
        assert w.pcg_kernel()[0] == "slab-batched"
        worlds.append(w)
    (x0, v0), (x1, v1) = (w.state(f64=True) for w in worlds)
    assert rel(x1, x0) <= 3e-7 and rel(v1, v0) <= 2e-4
    for i in range(count):
        a, b = worlds[1].body_stats(i), worlds[0].body_stats(i)
        assert abs(a["iterations"] - b["iterations"]) <= 1 and a["flags"] == b["flags"], (i, a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_steps_repeat_bit_for_bit_and_under_graph_replay(precision):
    for scene in (meshes.config1(), meshes.config2()):
        worlds = [SimWorld(scene, precision=precision) for _ in range(3)]
        worlds[2].set_graph(True)
        for _ in range(4):
            for w in worlds:
                w.step()
        x, v = worlds[0].state(f64=True)
        for w in worlds[1:]:
            np.testing.assert_array_equal(w.state(f64=True)[0], x)
            np.testing.assert_array_equal(w.state(f64=True)[1], v)
