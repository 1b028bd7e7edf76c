"""FP32 solves whose sums a float does not hold (GPU).

The reference adds its dot products in float: one that overflows ends the solve (no solution
from the first, a breakdown later), one that underflows counts as zero.  The kernels that add
in double must end such solves the same way: same flags and iterations as the kernel that adds
in float, and the same state (an overflow in the first sum leaves delta-v at zero, an underflow
converges at once).  Gravity sets the size: r.s of the first residual is about the mass times
(gravity dt)^2.
"""
import numpy as np
import pytest

from physik_b200 import meshes

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402

SHAPES = [(4, 3, 2), (17, 16, 15)]  # a cluster, all SMs


def step(shape, gravity, batched=False, **env):
    young = 1e5 if abs(gravity) > 1 else 1e-20  # (so soft that rounding leaves no force at rest)
    scene = meshes.small_box(*shape, young=young)
    if batched:
        scene.bodies += meshes.small_box(3, 4, 5, young=young, seed=4).bodies
    scene.gravity = (0.0, 0.0, gravity)
    with pytest.MonkeyPatch.context() as mp:
        for k, v in env.items():
            mp.setenv(k, v)
        w = SimWorld(scene, precision="fp32")
        w.set_batched(batched)
        w.step()
        return w.cg_stats(), w.state()


@pytest.mark.parametrize("env", [{}, {"PK_PCG_RESIDENT": "0"}], ids=["resident", "part"])
@pytest.mark.parametrize("gravity", [-1e23, -1e-24], ids=["overflow", "underflow"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_sums_end_the_solve_as_in_float(shape, gravity, env):
    (a, (xa, va)), (b, (xb, vb)) = step(shape, gravity, **env), step(shape, gravity, PK_PCG_KERNEL="plain")
    assert a["flags"] == b["flags"] and a["iterations"] == b["iterations"] == 0
    assert a["converged"] == b["converged"] == (1 if abs(gravity) < 1 else 0)
    np.testing.assert_array_equal(xa, xb)
    np.testing.assert_array_equal(va, vb)


@pytest.mark.parametrize("gravity", [-1e23, -1e-24], ids=["overflow", "underflow"])
def test_bodies_of_a_batch_end_the_same(gravity):
    a, b = step((4, 3, 2), gravity, True), step((4, 3, 2), gravity, True, PK_PCG_KERNEL="plain")
    assert a[0]["flags"] == b[0]["flags"] and a[0]["iterations"] == b[0]["iterations"] == 0
    for p, q in zip(a[1], b[1]):
        np.testing.assert_array_equal(p, q)


@pytest.mark.parametrize("env", [{}, {"PK_PCG_RESIDENT": "0"}], ids=["resident", "part"])
def test_a_large_solve_that_a_float_holds_is_solved(env):
    """r.s about 1e34: the other end of the same rule."""
    a, b = step((4, 3, 2), -3e18, **env), step((4, 3, 2), -3e18, PK_PCG_KERNEL="plain")
    assert a[0]["converged"] == b[0]["converged"] == 1 and a[0]["flags"] == b[0]["flags"]
    assert abs(a[0]["iterations"] - b[0]["iterations"]) <= 1
