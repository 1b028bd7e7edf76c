"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case is a world of Kuhn-split box bodies driven through the public entry points
(``SimWorld`` and the C ABI it wraps).  A pass uploads the bodies' positions and velocities
from pinned host memory, advances them and reads the new state back -- the end-to-end step
of the repository's benchmark -- so that every pass of a state does the same work.

kinds
    step      ``frames`` implicit steps of one soft body (one coupled block-Jacobi PCG a step)
    batch     one implicit step of many uneven independent bodies, one PCG per body, replayed
              as a CUDA graph
    explicit  one frame of ``substeps`` explicit substeps (no solve)
    adjoint   the backward pass of one implicit step (per-element Young's moduli)

The mesh families, materials, time steps, tolerances and iteration caps are those of the
repository's five benchmark workloads (``physik_b200/meshes.py``), over the range of sizes
that its tests and benchmark use.
"""
import ctypes
import math

import numpy as np
import torch

KUHN = np.array([[0, 1, 2, 6], [0, 2, 3, 6], [0, 3, 7, 6], [0, 7, 4, 6], [0, 4, 5, 6], [0, 5, 1, 6]])
CORNERS = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])
GRAVITY = (0.0, 0.0, -9.81)
DENSITY = 1000.0
MAX_CELLS = 128 * 64 * 64  # the largest listed body
L2_BYTES = 126e6


def _case(name, kind, cells, precision, h, young, poisson, dt, **more):
    c = {"name": name, "kind": kind, "nx": cells[0], "ny": cells[1], "nz": cells[2], "precision": precision, "h": h,
         "young": young, "poisson": poisson, "dt": dt, "frames": 1, "substeps": 1, "bodies": 1, "shape_seed": 0,
         "lo": 0, "hi": 0, "jitter": 0.05, "tolerance": 1e-6, "iterations": 100}
    c.update(more)
    return c


def _explicit_dt(h, young, poisson, substeps):
    """A frame of explicit substeps at a quarter of the smallest element's acoustic limit."""
    lam = young * poisson / ((1 + poisson) * (1 - 2 * poisson))
    mu = young / (2 * (1 + poisson))
    return 0.25 * h / math.sqrt((lam + 2 * mu) / DENSITY) * substeps


def listed():
    return [
        # the smallest thing one steps: an interactive prop of a few cells, one frame
        _case("box 4x3x2 mixed", "step", (4, 3, 2), "mixed", 0.1, 1e4, 0.3, 1 / 60, jitter=0.1),
        # the plain small cube in the reference's scalar type, a few frames between reads
        _case("cube 8 fp32", "step", (8, 8, 8), "fp32", 0.125, 1e5, 0.3, 1 / 60, jitter=0.1, frames=4),
        # the differentiable rollout's beam: its forward steps between checkpoints ...
        _case("beam 32x8x8 fp64", "step", (32, 8, 8), "fp64", 1 / 32, 1e5, 0.3, 1 / 60, jitter=0.0, frames=4,
              tolerance=1e-8, iterations=1024),
        # ... and one backward step of it
        _case("beam 32x8x8 adjoint", "adjoint", (32, 8, 8), "fp64", 1 / 32, 1e5, 0.3, 1 / 60, jitter=0.0,
              tolerance=1e-8, iterations=1024),
        # the single stiff beam in mixed precision, and its FP64 comparison run
        _case("beam 64x16x16 mixed", "step", (64, 16, 16), "mixed", 1 / 16, 1e6, 0.45, 1 / 120, jitter=0.0),
        _case("beam 64x16x16 fp64", "step", (64, 16, 16), "fp64", 1 / 16, 1e6, 0.45, 1 / 120, jitter=0.0),
        # a mid-size body with odd, uneven sides
        _case("block 61x47x29 mixed", "step", (61, 47, 29), "mixed", 1 / 47, 3e5, 0.4, 1 / 60),
        # an explicit frame of substeps (the reference's other integrator)
        _case("beam 64x16x16 explicit", "explicit", (64, 16, 16), "fp32", 1 / 16, 1e6, 0.3,
              _explicit_dt(1 / 16, 1e6, 0.3, 16), jitter=0.0, substeps=16),
        # many small props of a scene, one solve each
        _case("batch 96 small fp32", "batch", (0, 0, 0), "fp32", 0.05, 1e5, 0.35, 1 / 60, jitter=0.0, bodies=96,
              lo=2, hi=9, shape_seed=5),
        # the batched uneven bodies
        _case("batch 256 mixed", "batch", (0, 0, 0), "mixed", 0.05, 1e5, 0.35, 1 / 60, jitter=0.0, bodies=256,
              lo=4, hi=24, shape_seed=1),
        # the large body whose matrix is far larger than the caches, and its FP64 run
        _case("block 128x64x64 mixed", "step", (128, 64, 64), "mixed", 1 / 64, 5e5, 0.4, 1 / 60),
        _case("block 128x64x64 fp64", "step", (128, 64, 64), "fp64", 1 / 64, 5e5, 0.4, 1 / 60),
    ]


def _draw_cells(rng, lo, hi):
    """Three sides whose product is spread over the logarithm of [lo, hi]."""
    total = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(-0.45, 0.45), rng.uniform(-0.45, 0.45)
    base = total ** (1 / 3)
    sides = [max(2, round(base * math.exp(t))) for t in (a, b, -a - b)]
    while sides[0] * sides[1] * sides[2] > hi:
        sides[sides.index(max(sides))] -= 1
    return tuple(sides)


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "batch", "batch", "explicit", "adjoint"])
    young, poisson = math.exp(rng.uniform(math.log(3e4), math.log(1e6))), rng.uniform(0.25, 0.45)
    dt = 1 / rng.choice([60, 90, 120])
    if kind == "step":
        cells = _draw_cells(rng, 24, MAX_CELLS)
        small = cells[0] * cells[1] * cells[2] < 4000
        c = _case("", kind, cells, rng.choice(["mixed", "mixed", "fp32", "fp64"]), 1 / max(cells), young, poisson, dt,
                  jitter=rng.choice([0.0, 0.05, 0.1]), frames=rng.choice([1, 2, 4]) if small else 1)
    elif kind == "batch":
        hi = rng.randint(6, 24)
        bodies = max(8, int(256 * math.exp(-rng.uniform(0.0, 3.0))))
        c = _case("", kind, (0, 0, 0), rng.choice(["mixed", "mixed", "fp32"]), 0.05, young, poisson, dt, jitter=0.0,
                  bodies=bodies, lo=rng.randint(2, 4), hi=hi, shape_seed=rng.randrange(1 << 20))
    elif kind == "explicit":
        sub = rng.choice([4, 8, 16])
        cells = _draw_cells(rng, 200, 60000)
        h = 1 / max(cells)
        c = _case("", kind, cells, rng.choice(["fp32", "mixed", "fp64"]), h, young, poisson,
                  _explicit_dt(h, young, poisson, sub), substeps=sub)
    else:
        cells = _draw_cells(rng, 100, 6000)
        c = _case("", kind, cells, "fp64", 1 / max(cells), young, poisson, dt, tolerance=1e-8, iterations=1024)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _shapes(case):
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"])]
    rng = np.random.default_rng(case["shape_seed"])
    return [tuple(int(c) for c in s) for s in rng.integers(case["lo"], case["hi"] + 1, size=(case["bodies"], 3))]


def _grid(nx, ny, nz):
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    idx = np.stack([i.ravel(), j.ravel(), k.ravel()], 1)
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    corner = np.stack([i.ravel(), j.ravel(), k.ravel()], 1)[:, None] + CORNERS
    ids = corner[..., 0] + (nx + 1) * (corner[..., 1] + (ny + 1) * corner[..., 2])
    return idx, ids[:, KUHN].reshape(-1, 4).astype(np.int32)


def _inputs(case, seed):
    """Bodies (rest positions, tets, pinned nodes, material) and their moving state, float32."""
    rng = np.random.default_rng([seed, 77])
    bodies, xs, vs = [], [], []
    for nx, ny, nz in _shapes(case):
        idx, tets = _grid(nx, ny, nz)
        h = case["h"]
        rest = idx * h
        if case["jitter"] > 0:
            rest = rest + rng.uniform(-1, 1, rest.shape) * (case["jitter"] * h)
        rest = rest.astype(np.float32)
        pinned = idx[:, 0] == 0
        young, poisson = case["young"], case["poisson"]
        size = h * max(nx, ny, nz)
        c = rest - rest.mean(0)
        if case["kind"] == "batch":  # per-body material, a random pose and a rigid velocity
            young = math.exp(rng.uniform(math.log(1e4), math.log(1e6)))
            poisson = rng.uniform(0.25, 0.45)
            q = rng.normal(size=4) * (1, 0.2, 0.2, 0.2) + (2, 0, 0, 0)
            w, x, y, z = q / np.linalg.norm(q)
            rot = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                            [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                            [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])
            x0 = c @ rot.T + rest.mean(0)
            v0 = np.tile(rng.normal(0, 0.5, 3), (len(rest), 1))
        else:  # a bent, moving body
            amp, ph = rng.uniform(0.01, 0.02, 3) * size, rng.uniform(0, 2 * math.pi, 3)
            t = idx[:, :1] * (h / size)
            x0 = rest + amp * t * np.sin(1.5 * t + ph) + rng.uniform(-1, 1, rest.shape) * (1e-3 * h)
            v0 = t * rng.normal(0, 0.5, 3) + 0.2 * np.sin(3 * c[:, ::-1] / size + ph)
        v0 = np.where(pinned[:, None], 0.0, v0)
        tet_young = None
        if case["kind"] == "adjoint":
            tet_young = np.exp(rng.normal(math.log(young), 0.3, len(tets))).astype(np.float32)
        bodies.append((rest, tets, pinned, float(young), float(poisson), tet_young, (nx, ny, nz)))
        xs.append(x0)
        vs.append(v0)
    x = np.concatenate(xs).astype(np.float32)
    v = np.concatenate(vs).astype(np.float32)
    bars = None
    if case["kind"] == "adjoint":
        bars = rng.normal(size=(2,) + x.shape)
    return bodies, x, v, bars


def _pinned_copy(a, dtype):
    t = torch.empty(a.shape, dtype=dtype, pin_memory=True)
    t.numpy()[...] = a
    return t


# ------------------------------------------------------------------ the case as a program
def prepare(case, seed):
    from physik_b200 import _lib, meshes
    from physik_b200.world import SimWorld

    torch.cuda.init()
    bodies, x, v, bars = _inputs(case, seed)
    scene = meshes.Scene("case", [
        meshes.Body(rest, tets, pinned, density=DENSITY, young=young, poisson=poisson, tet_young=ty, cells=cells)
        for rest, tets, pinned, young, poisson, ty, cells in bodies], dt=case["dt"], steps=case["frames"],
        gravity=GRAVITY, tolerance=case["tolerance"], max_iterations=case["iterations"])
    world = SimWorld(scene, precision=case["precision"], implicit=case["kind"] != "explicit")
    api = _lib.PX
    api.PHYSIK_SetSubstepCount(world.h, case["substeps"])
    if case["kind"] == "batch":
        world.set_batched(True)
        world.set_graph(True)
    wide = case["precision"] == "fp64"
    dtype = torch.float64 if wide else torch.float32
    state = {"world": world, "api": api, "frames": case["frames"], "kind": case["kind"], "n": world.node_count,
             "set": api.PHYSIK_B200_SetNodeStatesF64 if wide else api.PHYSIK_B200_SetNodeStates,
             "get": api.PHYSIK_B200_GetNodeStatesF64 if wide else api.PHYSIK_B200_GetNodeStates,
             "x": _pinned_copy(x, dtype), "v": _pinned_copy(v, dtype),
             "x1": torch.empty(x.shape, dtype=dtype, pin_memory=True),
             "v1": torch.empty(x.shape, dtype=dtype, pin_memory=True)}
    for key in ("x", "v", "x1", "v1"):
        state["p" + key] = ctypes.c_void_p(state[key].data_ptr())
    if case["kind"] == "adjoint":
        state["xbar"], state["vbar"] = bars
    # The first frames of a program build the scene, upload it and capture the step.
    _set(state)
    for _ in range(3 if case["kind"] == "batch" else 1):
        world.step()
    world.synchronize()
    return state


def _set(s):
    if s["set"](s["world"].h, s["px"], s["pv"], s["n"]) < 0:
        raise RuntimeError("SetNodeStates: " + s["world"].error())


def run(s):
    w = s["world"]
    _set(s)
    if s["kind"] == "adjoint":
        theta = np.zeros(w.tet_count())
        xbar, vbar = w.adjoint_step(s["xbar"], s["vbar"], theta)
        return {"xbar": xbar, "vbar": vbar, "theta": theta}
    for _ in range(s["frames"]):
        w.step()
    if s["get"](w.h, s["px1"], s["pv1"], s["n"]) < 0:
        raise RuntimeError("GetNodeStates: " + w.error())
    return {"x": s["x1"], "v": s["v1"]}


# ------------------------------------------------------------------ what a pass cannot do without
def _counts(case):
    nodes = rows = tets = upper = 0
    for nx, ny, nz in _shapes(case):
        x, y, z = nx, ny + 1, nz + 1  # the x = 0 face is pinned
        nodes += (nx + 1) * y * z
        rows += x * y * z
        tets += 6 * nx * ny * nz
        # edges of the Kuhn grid between dynamic nodes: 3 axes, 3 face diagonals, the main diagonal
        upper += x * y * z + (x - 1) * y * z + x * (y - 1) * z + x * y * (z - 1) + (x - 1) * (y - 1) * z
        upper += (x - 1) * y * (z - 1) + x * (y - 1) * (z - 1) + (x - 1) * (y - 1) * (z - 1)
    return nodes, rows, tets, upper


def work(case):
    """Bytes: the state in and out, the tets' rest data, and the assembled system written and
    read; a matrix larger than the L2 cache is read again in every CG iteration.  Operations:
    about 600 a tet and 2 x 9 a block product, both triangles."""
    nodes, rows, tets, upper = _counts(case)
    real = 8 if case["precision"] == "fp64" else 4
    state = 12 * real * nodes
    rest = tets * (16 + 13 * real)
    if case["kind"] == "explicit":
        n = case["substeps"]
        return {"bytes": state + rest, "flops": n * 400.0 * tets}
    matrix = upper * (9 * real + 4) + rows * 12 * real
    # iterations of the workloads' solves: the cap for the stiff large bodies, fewer for small ones
    its = min(case["iterations"], 30 + 0.9 * max(max(s) for s in _shapes(case)))
    solves = 2 if case["kind"] == "adjoint" else case["frames"]
    reads = its if matrix > L2_BYTES else 1
    return {"bytes": state + case["frames"] * rest + solves * matrix * (1 + reads),
            "flops": case["frames"] * 600.0 * tets + solves * its * (36.0 * upper + 60.0 * rows)}


# ------------------------------------------------------------------ the same in 64 bits
class _Exact:
    """One world in float64, matrix free: every product goes tet by tet."""

    def __init__(self, case, seed):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f32 = lambda a: float(np.float32(a))  # noqa: E731  (the C ABI takes floats)
        bodies, x, v, bars = _inputs(case, seed)
        tets, rest, young, poisson, pinned, body, first = [], [], [], [], [], [], 0
        for i, (r, t, p, e, nu, ty, _) in enumerate(bodies):
            tets.append(t.astype(np.int64) + first)
            rest.append(r)
            young.append(np.full(len(t), f32(e)) if ty is None else ty.astype(np.float64))
            poisson.append(np.full(len(t), f32(nu)))
            pinned.append(p)
            body.append(np.full(len(r), i))
            first += len(r)
        put = lambda a: torch.from_numpy(np.concatenate(a)).to(dev)  # noqa: E731
        self.t, self.body, self.nb = put(tets), put(body), len(bodies)
        rest = put(rest).double()
        e, nu = put(young).double(), put(poisson).double()
        self.lam, self.mu = e * nu / ((1 + nu) * (1 - 2 * nu)), e / (2 * (1 + nu))
        dm = self.edges(rest)
        self.b = torch.linalg.inv(dm)
        self.vol = torch.linalg.det(dm).abs() / 6
        self.n = rest.shape[0]
        m = torch.zeros(self.n, dtype=torch.float64, device=dev)
        self.m = m.index_add_(0, self.t.reshape(-1), (f32(DENSITY) * self.vol / 4).repeat_interleave(4))[:, None]
        self.free = (~put(pinned)).double()[:, None]
        self.x, self.v = torch.from_numpy(x).to(dev).double(), torch.from_numpy(v).to(dev).double()
        self.bars = None if bars is None else torch.from_numpy(bars).to(dev)
        self.dt = float(np.float32(np.float32(case["dt"]) / np.float32(case["substeps"])))
        self.g = torch.tensor([f32(c) for c in GRAVITY], dtype=torch.float64, device=dev)
        self.tol, self.its = f32(case["tolerance"]), case["iterations"]

    def edges(self, x):
        p = x[self.t]
        return (p[:, 1:] - p[:, :1]).transpose(1, 2)

    def gather(self, q):
        """Sum over the tets of q times each corner's shape gradient, on the nodes."""
        h = (q @ self.b.transpose(1, 2)).transpose(1, 2)
        h = torch.cat([-h.sum(1, keepdim=True), h], 1)
        out = torch.zeros(self.n, 3, dtype=torch.float64, device=h.device)
        return out.index_add(0, self.t.reshape(-1), h.reshape(-1, 3))

    def rotations(self, f):
        r = f
        for _ in range(12):
            c0, c1, c2 = r[..., 0], r[..., 1], r[..., 2]
            cof = torch.stack([torch.linalg.cross(c1, c2), torch.linalg.cross(c2, c0), torch.linalg.cross(c0, c1)], -1)
            det = (c0 * cof[..., 0]).sum(-1)
            r = 0.5 * (r + cof / det[:, None, None])
        return r

    def stress(self, x):
        f = self.edges(x) @ self.b
        r = self.rotations(f)
        s = r.transpose(1, 2) @ f
        eps = 0.5 * (s + s.transpose(1, 2)) - torch.eye(3, dtype=torch.float64, device=f.device)
        return r, self.vol[:, None, None] * (r @ self.law(eps))

    def law(self, eps):
        tr = eps.diagonal(dim1=1, dim2=2).sum(1)
        return torch.diag_embed((self.lam * tr)[:, None].expand(-1, 3)) + 2 * self.mu[:, None, None] * eps

    def stiff(self, r, u):
        g = r.transpose(1, 2) @ self.edges(u) @ self.b
        return self.vol[:, None, None] * (r @ self.law(0.5 * (g + g.transpose(1, 2))))

    def dots(self, a, b):
        s = torch.zeros(self.nb, dtype=torch.float64, device=a.device)
        return s.index_add(0, self.body, (a * b).sum(1))

    def system(self):
        r, s = self.stress(self.x)
        dt = self.dt
        rhs = self.free * (dt * (self.m * self.g - self.gather(s)) - dt * dt * self.gather(self.stiff(r, self.v)))
        grads = torch.cat([-self.b.sum(1, keepdim=True), self.b], 1)
        p = grads @ r.transpose(1, 2)  # R g of the four corners
        gg = (grads * grads).sum(2)
        k = self.vol[:, None, None, None] * (
            (self.lam + self.mu)[:, None, None, None] * p[..., :, None] * p[..., None, :]
            + (self.mu[:, None] * gg)[..., None, None] * torch.eye(3, dtype=torch.float64, device=p.device))
        diag = torch.zeros(self.n, 9, dtype=torch.float64, device=p.device)
        diag = diag.index_add(0, self.t.reshape(-1), k.reshape(-1, 9)).reshape(-1, 3, 3) * (dt * dt)
        diag = diag + torch.diag_embed(self.m.expand(-1, 3))
        apply = lambda u: self.free * (self.m * u + dt * dt * self.gather(self.stiff(r, u)))  # noqa: E731
        return apply, torch.linalg.inv(diag), rhs

    def solve(self, apply, minv, b):
        x, r = torch.zeros_like(b), b
        s = (minv @ r[..., None])[..., 0]
        d, rho = s, self.dots(r, s)
        target = self.tol * self.tol * rho
        for _ in range(self.its):
            live = rho > target
            if not bool(live.any()):
                break
            q = apply(d)
            alpha = torch.where(live, rho / self.dots(d, q), 0.0)[self.body][:, None]
            x, r = x + alpha * d, r - alpha * q
            s = (minv @ r[..., None])[..., 0]
            new = self.dots(r, s)
            d = s + torch.where(live, new / rho, 0.0)[self.body][:, None] * d
            rho = torch.where(live, new, rho)
        return x

    def step(self):
        self.v = self.v + self.solve(*self.system())
        self.x = self.x + self.free * (self.dt * self.v)

    def step_explicit(self):
        a = self.free * (self.g - self.gather(self.stress(self.x)[1]) / self.m)
        self.v = self.v + self.dt * a
        self.x = self.x + self.free * (self.dt * self.v)

    def adjoint(self):
        apply, minv, rhs = self.system()
        du = self.solve(apply, minv, rhs)
        xb, vb = self.bars
        g = self.free * (vb + self.dt * xb)
        w = self.solve(apply, minv, g)
        z = self.v + du
        x = self.x.clone().requires_grad_(True)
        r, s = self.stress(x)
        wg = self.edges(w) @ self.b
        j = -(self.dt * s + self.dt * self.dt * self.stiff(r, z)) * wg
        j.sum().backward()
        vbar = torch.where(self.free > 0, g - apply(w) + self.m * w, vb)
        return {"xbar": xb + self.free * x.grad, "vbar": vbar, "theta": j.detach().sum((1, 2))}


def exact(case, seed):
    e = _Exact(case, seed)
    if case["kind"] == "adjoint":
        return e.adjoint()
    if case["kind"] == "explicit":
        for _ in range(case["substeps"]):
            e.step_explicit()
    else:
        for _ in range(case["frames"]):
            e.step()
    return {"x": e.x, "v": e.v}
