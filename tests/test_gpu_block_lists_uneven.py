"""Off-diagonal blocks whose lists differ within a warp (GPU).

A warp of the block-list kernel adds up 32 blocks' lists, of one tet or of many, some by the
short way and some by the long one, and its lanes then store each other's blocks.  A box joined
by a fan of 40 tets around one edge, every third tet so soft that it keeps its rotation and
stress (V mu below 1e-30), must give the blocks of the one-thread rows bit for bit, which share
nothing between lanes: every list is added in tet order in both.
"""
import numpy as np
import pytest

from physik_b200 import meshes

pytestmark = pytest.mark.gpu

pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402


def uneven_scene(seed):
    scene = meshes.small_box(6, 5, 4, seed=seed)
    box = scene.bodies[0]
    rng = np.random.default_rng(seed)
    n, fan = len(box.positions), 40
    angle = 0.12 * np.arange(fan + 1)
    ring = np.stack([np.cos(angle), np.sin(angle), 0.02 * np.arange(fan + 1)], axis=1) + [3.0, 0.0, 0.0]
    axis = np.array([[3.0, 0.0, -0.5], [3.0, 0.0, 0.5]])
    rest = np.concatenate([box.positions, axis, ring]).astype(np.float32)
    tets = np.concatenate([box.tets, [[n, n + 1, n + 2 + i, n + 3 + i] for i in range(fan)]]).astype(np.int32)
    pinned = np.concatenate([box.pinned, np.zeros(fan + 3, bool)])
    young = np.where(np.arange(len(tets)) % 3 == 0, 1e-30, 1e5).astype(np.float32)
    body = meshes.Body(rest, tets, pinned, density=1000.0, young=1e5, poisson=0.3, tet_young=young)
    body.initial_velocities = np.where(pinned[:, None], 0.0, rng.normal(0, 0.2, rest.shape)).astype(np.float32)
    scene.bodies = [body]
    return scene


@pytest.mark.parametrize("precision", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("seed", [1, 2])
def test_blocks_equal_the_thread_rows(precision, seed, monkeypatch):
    systems = []
    for rows in ("", "thread"):
        monkeypatch.setenv("PK_ROW_KERNEL", rows)
        w = SimWorld(uneven_scene(seed), precision=precision)
        w.step()
        systems.append(w.system())
    a, b = systems
    upper = np.ones(len(a["col"]), bool)
    upper[a["row_start"][:-1]] = False  # (rows of more than 16 blocks sum their diagonal in another order)
    assert np.abs(a["values"]).max() > 0
    np.testing.assert_array_equal(a["values"][upper], b["values"][upper])
