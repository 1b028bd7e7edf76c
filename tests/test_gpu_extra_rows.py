"""Point connections and host-emitted contributions added to the assembled rows (GPU), against a
dense assembly in 64 bits.

The soft bodies' part is the FP64 oracle's system; the masses, forces, blocks
(SolverData::AssembleImplicitMatrixAndRhs, SolverData.cpp:308-465) and connections
(PointConnection::UpdateSystem, PointConnection.cpp:55-140) are added to it with numpy on the
full 3n x 3n matrix.  With F = k (target - p) - c u of a connection's point p and velocity u,
corner a receives dt w_a F - dt^2 sum_b k w_a w_b v_b and the blocks dt^2 k w_a w_b I; an emitted
block adds -dt^2 B v_column to its row, and dt^2 B where both nodes are dynamic (a lower one only
where nothing emits its upper twin); an emitted mass adds m I and dt m g.

Tolerances: FP64 1e-12 of the largest entry (sums of some tens of terms of 1.1e-16, with room for
the shape gradients), 1e-10 for the inverses (3x3 blocks of condition below 100); FP32 storage
the same with 6e-8 in place of 1.1e-16, 6e-4.
"""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

L = pytest.importorskip("physik_b200._lib")
from physik_b200.world import SimWorld  # noqa: E402
from tests.test_contributions import attach_ours, emissions, exact_scene  # noqa: E402

CONNECTIONS = [  # nodes, weights, target, stiffness, damping
    ((3, 4, 5, 8), (0.25, 0.25, 0.25, 0.25), (0.5, 0.25, 0.125), 64.0, 0.5),
    ((7, 8, 3, 30), (0.5, 0.0, 0.25, 0.25), (0.0, 0.5, 0.25), 32.0, 0.0),  # joins the bodies; a weight of zero
    ((0, 1, 5, 4), (0.125, 0.375, 0.25, 0.25), (0.25, 0.0, 0.5), 16.0, 1.0),  # node 0 is fixed
    ((33, 34, 31, 35), (0.25, 0.25, 0.25, 0.25), (0.5, 0.5, 0.5), 0.0, 2.0),  # no stiffness: a force only
]


def moving_scene():
    scene = exact_scene()
    rng = np.random.default_rng(3)
    for b in scene.bodies:
        v = np.round(rng.normal(0, 0.3, b.positions.shape) * 64) / 64
        b.initial_velocities = np.where(b.pinned[:, None], 0.0, v).astype(np.float32)
    return scene


def dense(rs, col, values):
    n = len(rs) - 1
    full = np.zeros((n, 3, n, 3))
    for r in range(n):
        for k in range(rs[r], rs[r + 1]):
            block = np.asarray(values[k]).T  # column-major
            full[r, :, col[k], :] = block
            full[col[k], :, r, :] = block.T
    return full


def expected(scene, emitters, connections):
    ora = po.Oracle(scene, "f64", float_inputs=True)
    x, v = np.array(ora.x).reshape(-1, 3), np.array(ora.v).reshape(-1, 3)
    ora.step()
    s = ora.last_system()
    row, dt, g = np.asarray(s.node_to_dyn), float(np.float32(scene.dt)), np.float32(scene.gravity).astype(np.float64)
    full, rhs, nodes = dense(s.row_start, s.col, s.values), np.array(s.rhs).reshape(-1, 3), len(x)
    fem = {(r, int(c)) for r in range(len(s.row_start) - 1) for c in s.col[s.row_start[r]:s.row_start[r + 1]]}
    blocks = [a for _, items in emitters for kind, a in items if kind == "block" and max(a[0], a[1]) < nodes]
    twins = fem | {(row[a], row[b]) for a, b, _ in blocks}
    twins |= {(row[a], row[b]) for nd, w, _, k, _ in connections for a, p in zip(nd, w) for b, q in zip(nd, w)
              if k * p * q != 0}
    eye = np.eye(3)
    for nd, w, target, k, c in connections:
        nd, w = np.array(nd), np.array(w)
        force = k * (np.array(target) - w @ x[nd]) - c * (w @ v[nd])
        for a, wa in zip(nd, w):
            if row[a] < 0 or wa == 0:
                continue
            rhs[row[a]] += dt * wa * force
            for b, wb in zip(nd, w):
                rhs[row[a]] -= dt * dt * k * wa * wb * v[b]
                if row[b] >= 0:
                    full[row[a], :, row[b], :] += dt * dt * k * wa * wb * eye
    for _, items in emitters:
        for kind, a in items:
            if a[0] >= nodes or row[a[0]] < 0:
                continue
            r = row[a[0]]
            if kind == "mass" and a[1] > 0:
                full[r, :, r, :] += a[1] * eye
                rhs[r] += dt * a[1] * g
            elif kind == "force" and np.all(np.isfinite(a[1])):
                rhs[r] += dt * np.array(a[1])
            elif kind == "block" and a[1] < nodes:
                rhs[r] -= dt * dt * (a[2] @ v[a[1]])
                c = row[a[1]]
                if c < 0 or (r > c and (c, r) in twins):
                    continue
                full[r, :, c, :] += dt * dt * a[2]
                if r != c:
                    full[c, :, r, :] += dt * dt * a[2].T
    return full, rhs


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("what", ["connections", "emitted", "both"])
@pytest.mark.parametrize("rows", ["", "thread"])
def test_rows_equal_a_dense_assembly(rows, what, precision, monkeypatch):
    monkeypatch.setenv("PK_ROW_KERNEL", rows)
    scene = moving_scene()
    emitters = emissions(scene) if what != "connections" else []
    if emitters:  # a lower block whose upper twin the soft body emits: its right-hand side only
        emitters.append((1001, [("block", (5, 4, np.diag([0.5, 0.25, 0.125])))]))
    connections = CONNECTIONS if what != "emitted" else []
    w = SimWorld(scene, precision=precision)
    keep = attach_ours(w, emitters)  # noqa: F841  (callbacks stay alive)
    for c in connections:
        w.add_point_connection(*c)
    w.step()
    assert w.cg_stats()["flags"] & L.FLAG_INTEGRATED
    got = w.system()
    full, rhs = expected(scene, emitters, connections)
    assert len(rhs) == len(got["row_start"]) - 1
    tol = 1e-12 if precision == "fp64" else 6e-4
    assert np.abs(dense(got["row_start"], got["col"], got["values"]) - full).max() <= tol * np.abs(full).max()
    assert np.abs(got["rhs"] - rhs).max() <= tol * np.abs(rhs).max()
    inverse = np.array([np.linalg.inv(full[r, :, r, :]) for r in range(len(rhs))])
    bound = (1e-10 if precision == "fp64" else 6e-4) * np.abs(inverse).max()
    assert np.abs(np.transpose(got["minv"], (0, 2, 1)) - inverse).max() <= bound
