"""Batched solves on the streaming kernel (GPU): rounds, and the table the device builds for them.

Small bodies run on the resident kernel in clusters, so the batch tests that are about the
streaming kernel's rounds are repeated here with the resident kernel switched off, and with
the kernel asserted: bodies in several rounds of one launch against one-body oracles, the
round table from earlier iteration counts against a fresh one bit for bit, the batch kernel;
then many bodies on few blocks, under graph replay too.
"""
import numpy as np
import pytest

from tests import test_gpu_batch as batch

pytestmark = pytest.mark.gpu

pytest.importorskip("physik_b200._lib")
from physik_b200 import meshes  # noqa: E402
from physik_b200.world import SimWorld  # noqa: E402


class Streamed(SimWorld):
    def pcg_kernel(self):
        assert self.pcg_launched() in ("pcg_slab_kernel", "pcg_batch_kernel")
        return super().pcg_kernel()


@pytest.fixture(autouse=True)
def streaming(monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    monkeypatch.setattr(batch, "SimWorld", Streamed)


@pytest.mark.parametrize("blocks", [0, 2])
def test_rounds_match_one_body_worlds(blocks):
    batch.test_batched_part_resident_kernel_matches_one_body_worlds(blocks)


def test_the_round_table_does_not_change_results():
    batch.test_batched_round_table_does_not_change_results()


def test_it_agrees_with_the_batch_kernel(monkeypatch):
    batch.test_batched_part_resident_agrees_with_batch_kernel(monkeypatch)


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("count,blocks", [(40, 3), (200, 7), (200, 0)])
def test_many_bodies_on_few_blocks_repeat_under_graph_replay(count, blocks, precision):
    rng = np.random.default_rng(count)
    scene = meshes.small_box(*(int(c) for c in rng.integers(1, 7, 3)))
    for i in range(count - 1):
        scene.bodies += meshes.small_box(*(int(c) for c in rng.integers(1, 7, 3)), seed=i).bodies
    worlds = [SimWorld(scene, precision=precision) for _ in range(2)]
    for w in worlds:
        w.set_batched(True)
        if blocks:
            w.prepare(True)
            assert w.set_pcg_grid(blocks) > 0
    worlds[1].set_graph(True)
    for _ in range(4):  # the table of a step follows the counts of the one before
        for w in worlds:
            w.step()
    for w in worlds:
        assert w.pcg_launched() == "pcg_slab_kernel"
    for a, b in zip(*(w.state(f64=True) for w in worlds)):
        np.testing.assert_array_equal(a, b)
    assert [worlds[0].body_stats(i)["iterations"] for i in range(count)] == \
        [worlds[1].body_stats(i)["iterations"] for i in range(count)]
