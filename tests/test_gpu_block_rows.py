"""The assembled rows at the edges of the tet kernel's and the block kernel's tiles (GPU).

A fan of n tets around one edge: the two ends of the edge have rows of n + 3 blocks, every
tet is in both, and the block of the edge itself sums all n.  Sizes around one warp's records
(32 tets), one block's (64, 128), the lists' lanes (16), and a single tet.  Compared with the
FP64 oracle's assembled system (the reference's CPU assembly in double,
SolverData.cpp:308-465) and, for the explicit step, with the forces in that system's
right-hand side at rest velocity (dt (f + m g)).

Tolerances (FP64): a sum of at most 130 rounded terms is within 130 * 1.1e-16 = 1.5e-14 of
its terms' size; the shape gradients of a wedge of 1/20 rad lose a factor 20 on top and the
rotation as much, so 1e-12 of the largest entry, and 1e-10 for the inverse, whose 3x3 blocks'
condition stays below 100.  FP32: the same with 6e-8 for 1.1e-16, 6e-4.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from physik_b200 import meshes

pytestmark = pytest.mark.gpu

pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

SIZES = [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129]


def fan(n):
    angle = 0.05 * np.arange(n + 1) if n > 6 else 0.8 * np.arange(n + 1)
    ring = np.stack([np.cos(angle), np.sin(angle), 0.02 * np.arange(n + 1)], axis=1)
    rest = np.concatenate([[[0.0, 0.0, -0.5], [0.0, 0.0, 0.5]], ring]).astype(np.float32)
    tets = np.array([[0, 1, 2 + i, 3 + i] for i in range(n)], np.int32)
    rng = np.random.default_rng(n)
    body = meshes.Body(rest, tets, np.arange(n + 3) == n + 2, density=1000.0, young=1e5, poisson=0.3)
    moved = 1.02 * rest + rng.uniform(-1e-3, 1e-3, rest.shape)
    body.initial_positions = np.where(body.pinned[:, None], rest, moved).astype(np.float32)
    return meshes.Scene(f"fan{n}", [body], dt=1.0 / 60.0, steps=1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", SIZES)
def test_fan_rows_match_the_oracle(n, precision):
    scene = fan(n)
    rng = np.random.default_rng(n + 1000)
    speed = rng.normal(0, 0.2, (n + 3, 3)).astype(np.float32)
    speed[scene.bodies[0].pinned] = 0.0
    scene.bodies[0].initial_velocities = speed
    gpu = SimWorld(scene, precision=precision)
    ora = po.Oracle(scene, "f64", float_inputs=True)
    gpu.set_state(ora.x, ora.v, f64=True)
    gpu.step()
    ora.step()
    g, o = gpu.system(), ora.last_system()
    np.testing.assert_array_equal(g["row_start"], o.row_start)
    np.testing.assert_array_equal(g["col"], o.col)
    for key, tol in (("values", 1e-12), ("rhs", 1e-12), ("minv", 1e-10)):
        want = getattr(o, key)
        bound = (tol if precision == "fp64" else 6e-4) * np.abs(want).max()
        assert np.abs(g[key] - want).max() <= bound, key


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", SIZES)
def test_fan_explicit_step_matches_the_oracles_forces(n, precision):
    scene = fan(n)
    body = scene.bodies[0]
    ora = po.Oracle(scene, "f64", float_inputs=True)
    x0 = np.array(ora.x, np.float64).reshape(-1, 3)
    ora.step()  # from rest: its right-hand side is dt (f + m g)
    edges = body.positions.astype(np.float64)[body.tets]
    volume = np.abs(np.linalg.det(edges[:, 1:] - edges[:, :1])) / 6.0
    mass = np.zeros(n + 3)
    np.add.at(mass, body.tets.ravel(), np.repeat(body.density * volume / 4.0, 4))
    want = np.zeros((n + 3, 3))
    want[~body.pinned] = np.asarray(ora.last_system().rhs).reshape(-1, 3) / mass[~body.pinned, None]
    gpu = SimWorld(scene, precision=precision, implicit=False)
    gpu.set_state(x0, np.zeros_like(x0), f64=True)
    gpu.step()
    v = np.asarray(gpu.state(f64=True)[1], np.float64).reshape(-1, 3)
    assert np.abs(v - want).max() <= (1e-12 if precision == "fp64" else 6e-4) * np.abs(want).max()
