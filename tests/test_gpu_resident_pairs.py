"""The resident PCG kernel with blocks in tensor memory (GPU): two rows a thread in FP32 (parts
of more than 256 rows), one in FP64 (parts whose blocks exceed registers and shared memory).

The launch is limited to a few blocks, so that small boxes reach these parts: up to the most
rows of a block (640), one block alone, several with a ragged last part; then a box over all
SMs.  One teacher-forced step from the same state is compared with the FP64 oracle with the
tolerances of the other resident tests (test_gpu_resident.py).
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

TOL = {"fp64": (1e-14, 1e-12), "mixed": (3e-7, 2e-4), "fp32": (3e-7, 2e-4)}
# box, blocks of the launch (0: all), precision
CASES = [((10, 7, 7), 1, "mixed"), ((9, 7, 7), 1, "fp32"), ((23, 7, 7), 3, "mixed"), ((17, 8, 8), 3, "mixed"),
         ((29, 7, 7), 3, "fp32"), ((41, 9, 9), 7, "mixed"), ((47, 29, 29), 0, "mixed"),
         ((9, 8, 8), 3, "fp64"), ((10, 8, 8), 4, "fp64"), ((12, 10, 8), 5, "fp64"), ((41, 29, 29), 0, "fp64")]


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("shape,blocks,precision", CASES, ids=lambda c: str(c).replace(", ", "x"))
def test_parts_in_tensor_memory_follow_the_fp64_oracle(shape, blocks, precision):
    scene = meshes.small_box(*shape)
    gpu = SimWorld(scene, precision=precision)
    if blocks:
        gpu.prepare(True)  # the limit belongs to the uploaded scene
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
        assert rel(x, ora.x) <= TOL[precision][0]
        assert rel(v, ora.v) <= TOL[precision][1]
        assert abs(st["iterations"] - ora.last_stats()["iterations"]) <= 1
