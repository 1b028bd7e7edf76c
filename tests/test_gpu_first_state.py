"""A first state that is not finite (GPU): no step of it integrates, and it leaves no trace.

The layouts of the resident and part-resident kernels are cut by the first positions.  A world
whose first positions hold a NaN or an infinity reports a step that did not integrate; after a
finite state is set it follows the FP64 oracle with the tolerances of test_gpu_resident.py, and
where the finite state comes before the first step, bit for bit with a world that never held
another.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

TOL = {"fp64": (1e-14, 1e-12), "mixed": (3e-7, 2e-4)}


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("resident", ["1", "0"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bad", [np.nan, np.inf], ids=str)
def test_a_step_from_it_fails_and_the_next_state_is_solved(bad, precision, resident, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", resident)
    scene = meshes.small_box(13, 9, 7)
    w = SimWorld(scene, precision=precision)
    ora = po.Oracle(scene, "f64", float_inputs=True)
    x = np.array(ora.x, np.float64).reshape(-1, 3)
    x[1::5, 0] = bad
    w.set_state(x, np.zeros_like(x), f64=True)
    w.step()
    assert not w.cg_stats()["flags"] & L.FLAG_INTEGRATED
    for _ in range(2):
        w.set_state(ora.x, ora.v, f64=True)
        w.step()
        ora.step()
        got = w.state(f64=True)
        assert w.cg_stats()["flags"] & L.FLAG_INTEGRATED
        assert rel(got[0], ora.x) <= TOL[precision][0] and rel(got[1], ora.v) <= TOL[precision][1]


@pytest.mark.parametrize("resident", ["1", "0"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_finite_state_before_the_first_step_decides_the_layout(precision, resident, monkeypatch):
    monkeypatch.setenv("PK_PCG_RESIDENT", resident)
    scene = meshes.small_box(13, 9, 7)
    plain, other = SimWorld(scene, precision=precision), SimWorld(scene, precision=precision)
    x, v = plain.state(f64=True)
    plain.prepare(True)
    plain.set_state(x, v, f64=True)
    broken = np.array(x)
    broken[1::5, 0] = np.nan
    other.set_state(broken, v, f64=True)
    other.prepare(True)  # the scene and this state go to the device
    other.set_state(x, v, f64=True)
    for w in (plain, other):
        w.step()
        assert w.cg_stats()["flags"] & L.FLAG_INTEGRATED
    for a, b in zip(plain.state(f64=True), other.state(f64=True)):
        np.testing.assert_array_equal(a, b)
