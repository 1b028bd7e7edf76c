"""Which PCG kernel a solve launches (GPU), by the name of its function.

``pcg_kernel`` keeps its numbers, several of which stand for more than one kernel; the scenes
that the kernels' own tests step must run on those kernels, in every precision and with the
launch limits that those tests set, also batched and replayed as a graph.
"""
import pytest

from physik_b200 import meshes

pytestmark = pytest.mark.gpu

pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402
from tests import test_gpu_part, test_gpu_resident, test_gpu_resident_pairs, test_gpu_slab64  # noqa: E402

RES, PART, SLAB, RING = "pcg_res_kernel", "pcg_part_kernel", "pcg_slab_kernel", "pcg_ring_kernel"


def launched(scene, precision, blocks=0, batched=False, graph=False):
    w = SimWorld(scene, precision=precision)
    assert w.pcg_launched() == ""
    if batched:
        w.set_batched(True)
    if graph:
        w.set_graph(True)
    if blocks:
        w.prepare(True)
        assert w.set_pcg_grid(blocks) > 0
    for _ in range(3 if graph else 1):
        w.step()
    return w.pcg_launched()


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("shape", test_gpu_resident.SHAPES, ids=str)
def test_boxes_that_fit_the_chip_are_resident(shape, precision):
    assert launched(meshes.small_box(*shape), precision) == RES


@pytest.mark.parametrize("shape,blocks,precision", test_gpu_resident_pairs.CASES, ids=str)
def test_parts_in_tensor_memory_are_resident(shape, blocks, precision):
    assert launched(meshes.small_box(*shape), precision, blocks) == RES


@pytest.mark.parametrize("precision,cases", [("fp64", test_gpu_slab64.CASES), ("mixed", test_gpu_part.CASES),
                                             ("fp32", test_gpu_part.CASES)], ids=["fp64", "mixed", "fp32"])
def test_streamed_systems_run_on_the_part_kernel(precision, cases, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", "0")
    for shape, blocks in cases:
        assert launched(meshes.small_box(*shape), precision, blocks) == PART, shape


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_workloads_and_graph_replay(precision):
    for scene in (meshes.config1(), meshes.config2()):
        assert launched(scene, precision, graph=True) == RES


@pytest.mark.parametrize("resident,kernel", [("1", RES), ("0", SLAB)])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_batches(precision, resident, kernel, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", resident)
    scene = meshes.small_box(5, 4, 3)
    scene.bodies += meshes.small_box(6, 3, 4, seed=2).bodies
    assert launched(scene, precision, batched=True) == kernel


@pytest.mark.parametrize("env,kernel", [({"PK_PCG_KERNEL": "ring"}, RING), ({"PK_PCG_KERNEL": "staged"}, "pcg_kernel"),
                                        ({"PK_PCG_KERNEL": "plain"}, "pcg_kernel"),
                                        ({"PK_SLAB_FORM": "sym"}, SLAB)], ids=str)
def test_requested_kernels(env, kernel, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    assert launched(meshes.small_box(9, 9, 9), "mixed") == kernel


def test_fp64_batches_run_on_the_batch_kernel():
    scene = meshes.small_box(5, 4, 3)
    scene.bodies += meshes.small_box(6, 3, 4, seed=2).bodies
    assert launched(scene, "fp64", batched=True) == "pcg_batch_kernel"
