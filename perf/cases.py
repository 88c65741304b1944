"""Performance cases of the VBD framework: what a program that uses it has it do, through its public
entry points, over the range of sizes and options it is used with.

The kinds:

* ``step``: one time step of one mesh (``pbat.gpu.vbd.Integrator.step``), the simulation loop of every
  single-object program; plain VBD or Chebyshev, with damping and substeps.
* ``batch``: one time step of many meshes of uneven size (``BatchedIntegrator.step``).
* ``rollout``: a differentiable rollout, forward and backward (``pbat.gpu.vbd.rollout``), as
  trajectory optimisation runs it: the gradient of the end state's distance to a target with respect to
  the initial positions and velocities, of a body whose stiffness varies over it.
* ``contact``: one time step of cubes hitting a fixed slab (surface mesh, bodies, contact parameters), from
  the moment before they touch, as a planner that tries one state again and again steps it.
* ``bvh``: a hierarchy over the triangle boxes of a surface and the nearest triangle of every query point
  (``pbat.gpu.geometry.Bvh``), from host arrays.

Without contact a time step goes on from the state the last one left, as a simulation does; positions and velocities are
read into device tensors after it (``pbgb_vbd_get_positions_device``, ``_velocities_device``).  Meshes are
caught in mid-motion: a swing about the pinned face or a fall of a few metres per second, with a small
random velocity on top.
"""

from __future__ import annotations

import ctypes as C
import itertools

import numpy as np
import torch

from physicsbasedanimationtoolkit_gb300 import _capi, pbat

DT = 1.0 / 60.0
G = np.array([0.0, 0.0, -9.81])


def listed():
    return [
        # The smallest mesh a program steps: 27 vertices, all latency and launches.
        dict(name="step_2x2x2", kind="step", nx=2, ny=2, nz=2, iterations=20, substeps=1, rho=0.0, kD=0.0, strategy=4),
        # The unit cube of the tests: 1331 vertices, 20 plain iterations, the default initial guess.
        dict(name="step_10x10x10", kind="step", nx=10, ny=10, nz=10, iterations=20, substeps=1, rho=0.0, kD=0.0, strategy=4),
        # An odd-sized beam with Chebyshev acceleration, Rayleigh damping and substeps.
        dict(name="step_41x11x9_damped", kind="step", nx=41, ny=11, nz=9, iterations=15, substeps=2, rho=0.8, kD=1e-4, strategy=2),
        # A detailed single object, as large as the largest mesh of the batch benchmark.
        dict(name="step_32x32x32", kind="step", nx=32, ny=32, nz=32, iterations=20, substeps=1, rho=0.0, kD=0.0, strategy=4),
        # The benchmark's beam: 270,641 vertices, 50 Chebyshev iterations.
        dict(name="step_160x40x40", kind="step", nx=160, ny=40, nz=40, iterations=50, substeps=1, rho=0.95, kD=0.0, strategy=2),
        # Many small environments stepped together, as a learning loop does.
        dict(name="batch_48_small", kind="batch", meshes=48, nmin=2, nmax=7, iterations=20, rho=0.0),
        # The benchmark's batch of uneven cubes (6 to 32 hexes a side), fewer of them.
        dict(name="batch_64", kind="batch", meshes=64, nmin=6, nmax=32, iterations=20, rho=0.0),
        # The smallest differentiable rollout of the tests, checkpoints inside it.
        dict(name="rollout_8x2x2", kind="rollout", nx=8, ny=2, nz=2, iterations=10, steps=4, every=2, rho=0.0, kD=0.0),
        # The differentiation beam (4961 vertices, 20 iterations), taped whole.
        dict(name="rollout_40x10x10", kind="rollout", nx=40, ny=10, nz=10, iterations=20, steps=5, every=5, rho=0.0, kD=0.0),
        # Cubes hitting a slab (active set, contact lists, contact terms in the sweep): a few coarse
        # ones, and a scene like the benchmark's.
        dict(name="contact_4_cubes", kind="contact", cubes=2, hexes=6, slab=16, iterations=20),
        dict(name="contact_9_cubes", kind="contact", cubes=3, hexes=11, slab=40, iterations=30),
        # Nearest triangles of 22,000 points on a surface of 43,000 triangles.
        dict(name="bvh_43k", kind="bvh", nu=147, nv=147),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["step", "step", "step", "step", "batch", "batch", "rollout", "rollout", "contact", "bvh"])
    if kind == "step":
        # From tens of vertices to two hundred thousand, beams and blocks.
        n = np.exp(rng.uniform(np.log(30.0), np.log(2.0e5)))
        aspect = rng.uniform(1.0, 4.0)
        side = (n / aspect) ** (1.0 / 3.0)
        cheb = rng.random() < 0.5
        return dict(kind="step", nx=max(2, int(side * aspect)), ny=max(2, int(side * rng.uniform(0.8, 1.2))),
                    nz=max(2, int(side)), iterations=rng.randint(10, 50 if cheb else 30), substeps=rng.choice([1, 1, 2]),
                    rho=round(rng.uniform(0.7, 0.9), 3) if cheb else 0.0, kD=rng.choice([0.0, 1e-4]),
                    strategy=rng.choice([2, 4]))
    if kind == "batch":
        nmin = rng.randint(2, 8)
        return dict(kind="batch", meshes=_log_int(rng, 6, 60), nmin=nmin, nmax=nmin + rng.randint(2, 22),
                    iterations=rng.randint(10, 20), rho=rng.choice([0.0, 0.0, 0.9]))
    if kind == "rollout":
        b = rng.randint(2, 9)
        return dict(kind="rollout", nx=b * rng.randint(2, 4), ny=b, nz=rng.randint(2, b + 1), iterations=rng.randint(8, 20),
                    steps=rng.randint(2, 5), every=rng.choice([2, 5]), rho=rng.choice([0.0, 0.85]), kD=0.0)
    if kind == "contact":
        h = _log_int(rng, 3, 11)
        return dict(kind="contact", cubes=rng.randint(1, 3), hexes=h, slab=rng.randint(2 * h, 4 * h), iterations=rng.randint(10, 30))
    n = _log_int(rng, 20, 140)
    return dict(kind="bvh", nu=n, nv=n + rng.randint(1, 9))


# ---- meshes -----------------------------------------------------------------------------------------


def _f32(a):
    """Rounded to FP32, so that the problem is the same in either precision."""
    return np.asarray(a, dtype=np.float32).astype(np.float64)


def _grid(nx, ny, nz, size):
    """Vertices and tets of an nx x ny x nz hex grid, each hex split into 6 tets along its main diagonal."""
    axes = [np.linspace(0.0, s, n + 1) for s, n in zip(size, (nx, ny, nz))]
    Z, Y, X = np.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    P = np.stack([X.ravel(), Y.ravel(), Z.ravel()], axis=1)
    k, j, i = (a.ravel() for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    T = np.empty((i.size, 6, 4), dtype=np.int64)
    for t, perm in enumerate(itertools.permutations(range(3))):
        corner, path = [0, 0, 0], [(0, 0, 0)]
        for axis in perm:
            corner[axis] = 1
            path.append(tuple(corner))
        even = perm in ((0, 1, 2), (1, 2, 0), (2, 0, 1))
        for a, (bx, by, bz) in enumerate(path if even else [path[0], path[2], path[1], path[3]]):
            T[:, t, a] = (i + bx) + (nx + 1) * ((j + by) + (ny + 1) * (k + bz))
    return P, T.reshape(-1, 4)


def _surface(T):
    """Outward boundary triangles."""
    faces = T[:, np.array([[1, 2, 3], [0, 3, 2], [0, 1, 3], [0, 2, 1]])].reshape(-1, 3)
    _, inverse, count = np.unique(np.sort(faces, axis=1), axis=0, return_inverse=True, return_counts=True)
    return faces[count[inverse.ravel()] == 1]


def _lame(E, nu):
    return E / (2.0 * (1.0 + nu)), E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))


def _block(nx, ny, nz, rng, E, nu, spread=0.0, size=None):
    """A jittered block or beam, pinned at x = 0 and swinging about that face."""
    size = size or (float(nx) / max(ny, nz), float(ny) / max(ny, nz), float(nz) / max(ny, nz))
    X, T = _grid(nx, ny, nz, size)
    pinned = np.nonzero(X[:, 0] == 0.0)[0]
    X = _f32(X + rng.uniform(-0.01, 0.01, X.shape) * (size[2] / nz))
    reach = X[:, 0] / size[0]
    v = np.stack([0.0 * reach, rng.uniform(-1, 1) * reach, -rng.uniform(2.0, 4.0) * reach], axis=1)
    v = _f32(v + rng.uniform(-0.1, 0.1, X.shape))
    v[pinned] = 0.0
    Ee = E * np.exp(spread * rng.standard_normal(T.shape[0]))
    mu, lam = _lame(Ee, nu)
    return dict(X=X, T=T, v=v, pinned=pinned, mu=mu, lam=lam, rho=np.full(T.shape[0], 1000.0))


def _meshes(case, seed):
    """The meshes of a step, batch or rollout case."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        # The sides come from the case, spread evenly over its range; materials and motion from the seed.
        n, lo, hi = case["meshes"], case["nmin"], case["nmax"]
        sides = [lo + ((b * 7919) % n) * (hi - lo + 1) // n for b in range(n)]
        return [_block(s, s, s, rng, float(np.exp(rng.uniform(np.log(1e5), np.log(1e7)))), float(rng.uniform(0.30, 0.48)),
                       size=(1.0, 1.0, 1.0)) for s in sides]
    if kind == "rollout":
        return [_block(case["nx"], case["ny"], case["nz"], rng, 1e5, 0.4, spread=0.3)]
    return [_block(case["nx"], case["ny"], case["nz"], rng, 5e5 if case.get("rho") else 1e6, 0.48 if case.get("rho") else 0.45)]


def _data(m, case):
    d = (pbat.sim.vbd.Data().with_volume_mesh(m["X"].T, m["T"].T).with_velocity(m["v"].T)
         .with_material(m["rho"], m["mu"], m["lam"]).with_dirichlet_vertices(m["pinned"]))
    if "strategy" in case:
        d = d.with_initialization_strategy(case["strategy"])
    elif case["kind"] == "rollout":
        d = d.with_initialization_strategy(2)
    if case.get("rho"):
        d = d.with_chebyshev_acceleration(case["rho"])
    if case.get("kD"):
        d = d.with_rayleigh_damping(case["kD"])
    return d


def _contact_scene(case, seed):
    """cubes x cubes blocks, each turned about the vertical, just above a fixed slab and falling on it."""
    rng = np.random.default_rng(seed)
    side, n = case["cubes"], case["slab"]
    Xs, Ts = _grid(n, n, 2, (float(side), float(side), 0.2))
    Xs = Xs - np.array([0.0, 0.0, 0.2])
    X, T, B, v = [Xs], [Ts], [np.zeros(Xs.shape[0], np.int64)], [np.zeros_like(Xs)]
    Xc, Tc = _grid(case["hexes"], case["hexes"], case["hexes"], (0.6, 0.6, 0.6))
    at = Xs.shape[0]
    for k in range(side * side):
        yaw = rng.uniform(0.0, 2.0 * np.pi)
        c, s = np.cos(yaw), np.sin(yaw)
        R = np.array([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]])
        place = np.array([k % side + 0.5, k // side + 0.5, rng.uniform(0.002, 0.01)])
        X.append((Xc - np.array([0.3, 0.3, 0.0])) @ R.T + place)
        T.append(Tc + at)
        B.append(np.full(Xc.shape[0], k + 1))
        v.append(np.tile([rng.uniform(-1, 1), rng.uniform(-1, 1), -rng.uniform(1.5, 2.5)], (Xc.shape[0], 1)))
        at += Xc.shape[0]
    X, T, v = _f32(np.vstack(X)), np.vstack(T), _f32(np.vstack(v))
    F = _surface(T)
    mu, lam = _lame(np.full(T.shape[0], 1e6), 0.45)
    return (pbat.sim.vbd.Data().with_volume_mesh(X.T, T.T).with_surface_mesh(np.unique(F), F.T)
            .with_bodies(np.concatenate(B)).with_velocity(v.T).with_material(np.full(T.shape[0], 1000.0), mu, lam)
            .with_dirichlet_vertices(np.arange(Xs.shape[0])).with_contact_parameters(1e6, 0.3, 1e-3)
            .with_initialization_strategy(2).construct())


def _sheet(case, seed):
    """A folded sheet: its vertices, its triangles and query points near it, one per vertex."""
    rng = np.random.default_rng(seed)
    nu, nv = case["nu"], case["nv"]
    u, w = np.meshgrid(np.linspace(0.0, 1.0, nu + 1), np.linspace(0.0, 1.0, nv + 1), indexing="ij")
    p, q = rng.uniform(0, 2 * np.pi, 2)
    P = np.stack([u + 0.04 * np.sin(24 * w + p), w, 0.05 * np.sin(18 * u + q) * np.cos(15 * w)], axis=-1).reshape(-1, 3)
    P = P + rng.uniform(-0.1, 0.1, P.shape) / nu
    i, j = (a.ravel() for a in np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij"))
    a, b, c, d = i * (nv + 1) + j, (i + 1) * (nv + 1) + j, (i + 1) * (nv + 1) + j + 1, i * (nv + 1) + j + 1
    F = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)])
    Q = P + 0.02 * rng.standard_normal(P.shape)
    return P.astype(np.float32), F, np.ascontiguousarray(Q.astype(np.float32).T)


# ---- the cases --------------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "bvh":
        P, F, s["points"] = _sheet(case, seed)
        s["V"], s["F"] = np.ascontiguousarray(P.T), np.ascontiguousarray(F.T)
        s["min"], s["max"] = s["V"].min(axis=1), s["V"].max(axis=1)
        s["boxes"] = pbat.gpu.geometry.Aabb()
        s["bvh"] = pbat.gpu.geometry.Bvh(F.shape[0])
        return s
    if kind == "contact":
        d = _contact_scene(case, seed)
        I = pbat.gpu.vbd.Integrator(d)
        s["x0"], s["v0"] = (torch.tensor(np.ascontiguousarray(a.T), dtype=torch.float32, device="cuda") for a in (d.x, d.v))
    elif kind == "batch":
        I = pbat.gpu.vbd.BatchedIntegrator([_data(m, case).construct() for m in _meshes(case, seed)])
    else:
        m = _meshes(case, seed)[0]
        I = pbat.gpu.vbd.Integrator(_data(m, case).construct())
        if kind == "rollout":
            f32 = dict(dtype=torch.float32, device="cuda")
            s["mu"], s["lam"] = torch.tensor(m["mu"]), torch.tensor(m["lam"])
            s["x0"] = torch.tensor(m["X"], **f32).requires_grad_()
            s["v0"] = torch.tensor(m["v"], **f32).requires_grad_()
            s["target"] = torch.tensor(m["X"], **f32)
    s["integrator"] = I
    s["x"], s["v"] = (torch.empty((I.n_vertices, 3), dtype=torch.float32, device="cuda") for _ in range(2))
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "bvh":
        b = state["bvh"]
        state["boxes"].construct(state["V"], state["F"])
        b.build(state["boxes"], state["min"], state["max"])
        return b.point_triangle_nearest_neighbours(state["boxes"], state["points"], state["V"], state["F"])
    I = state["integrator"]
    if case["kind"] == "rollout":
        for k in ("x0", "v0"):
            state[k].grad = None
        x, v = pbat.gpu.vbd.rollout(I, state["mu"], state["lam"], state["x0"], state["v0"], dt=DT,
                                    iterations=case["iterations"], steps=case["steps"], checkpoint_every=case["every"])
        loss = ((x - state["target"]) ** 2).sum()
        loss.backward()
        return dict(x=x.detach(), v=v.detach(), dx0=state["x0"].grad, dv0=state["v0"].grad)
    L = _capi.lib()
    if case["kind"] == "contact":
        _capi.check(L.pbgb_vbd_set_positions_device(I.handle, C.c_void_p(state["x0"].data_ptr())), I.handle)
        _capi.check(L.pbgb_vbd_set_velocities_device(I.handle, C.c_void_p(state["v0"].data_ptr())), I.handle)
    I.step(DT, case["iterations"], case.get("substeps", 1))
    _capi.check(L.pbgb_vbd_get_positions_device(I.handle, C.c_void_p(state["x"].data_ptr())), I.handle)
    _capi.check(L.pbgb_vbd_get_velocities_device(I.handle, C.c_void_p(state["v"].data_ptr())), I.handle)
    return dict(x=state["x"], v=state["v"])


def _counts(case):
    """(vertices, tets) of a case's meshes."""
    if case["kind"] == "batch":
        n, lo, hi = case["meshes"], case["nmin"], case["nmax"]
        sides = [lo + ((b * 7919) % n) * (hi - lo + 1) // n for b in range(n)]
        return sum((s + 1) ** 3 for s in sides), sum(6 * s**3 for s in sides)
    if case["kind"] == "contact":
        k, h, n = case["cubes"] ** 2, case["hexes"], case["slab"]
        return k * (h + 1) ** 3 + 3 * (n + 1) ** 2, k * 6 * h**3
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz


def work(case):
    """A step reads the state (positions, velocities, accelerations, masses) and the mesh (indices, two
    material words and a rest volume per tet, rest positions) once and writes the state once; an incidence
    costs about 50 FP32 operations an iteration.  A rollout does that per step and as much again, with
    about four times the operations, for its reverse.  A hierarchy reads the triangles, writes and reads a box per node, and answers one number a point."""
    if case["kind"] == "bvh":
        n, q = 2 * case["nu"] * case["nv"], (case["nu"] + 1) * (case["nv"] + 1)
        return dict(bytes=n * (12.0 + 2 * 2 * 24.0) + q * (12.0 + 12.0 + 4.0), flops=40.0 * q * np.log2(n))
    nv, nt = _counts(case)
    one = dict(bytes=nv * (40.0 + 12.0 + 24.0) + nt * 28.0, flops=4.0 * nt * 50.0 * case["iterations"] * case.get("substeps", 1))
    if case["kind"] == "rollout":
        return dict(bytes=2.0 * case["steps"] * one["bytes"], flops=5.0 * case["steps"] * one["flops"])
    return one


# ---- the same computation in 64 bits ----------------------------------------------------------------


def _colours(X, T, pinned):
    """Greedy colouring of the vertex graph: vertices by decreasing degree, each takes the least used
    colour that no neighbour has, the lowest one on a tie.  Returns the free vertices of every colour."""
    n = X.shape[0]
    e = np.concatenate([T[:, [a, b]] for a in range(4) for b in range(4) if a != b])
    key = np.unique(e[:, 0] * n + e[:, 1])
    src, dst = key // n, (key % n).tolist()
    ptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    order = np.argsort(-np.diff(ptr), kind="stable").tolist()
    ptr = ptr.tolist()
    colour, used = [-1] * n, []
    for u in order:
        taken = {colour[w] for w in dst[ptr[u]:ptr[u + 1]]}
        best = -1
        for c, k in enumerate(used):
            if c not in taken and (best < 0 or k < used[best]):
                best = c
        if best < 0:
            best = len(used)
            used.append(0)
        colour[u] = best
        used[best] += 1
    colour = np.array(colour)
    colour[pinned] = -1
    return [np.nonzero(colour == c)[0] for c in range(len(used))]


class _Exact:
    """VBD time steps of one system (several meshes side by side) in FP64 torch, differentiable."""

    def __init__(self, meshes, case):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        off = np.cumsum([0] + [m["X"].shape[0] for m in meshes])
        X = np.concatenate([m["X"] for m in meshes])
        T = np.concatenate([m["T"] + o for m, o in zip(meshes, off)])
        per = [[c + o for c in _colours(m["X"], m["T"], m["pinned"])] for m, o in zip(meshes, off)]
        colours = [np.concatenate(p) for p in itertools.zip_longest(*per, fillvalue=np.zeros(0, np.int64))]
        self.X, self.T = self.t(X), torch.as_tensor(T, device=self.dev)
        e = X[T[:, 1:]] - X[T[:, :1]]
        vol = np.linalg.det(e) / 6.0
        rho = np.concatenate([m["rho"] for m in meshes])
        self.m = self.t(np.bincount(T.ravel(), np.repeat(rho * vol / 4.0, 4), minlength=X.shape[0]))
        grads = np.linalg.inv(e).transpose(0, 2, 1)
        self.vol, self.grads = self.t(vol), self.t(np.concatenate([-grads.sum(1, keepdims=True), grads], axis=1))
        a = np.tile(G, (X.shape[0], 1))
        a[np.concatenate([m["pinned"] + o for m, o in zip(meshes, off)])] = 0.0
        self.a = self.t(a)
        corner = np.argsort(T.ravel(), kind="stable")
        ptr = np.concatenate([[0], np.cumsum(np.bincount(T.ravel(), minlength=X.shape[0]))])
        self.sets = []
        for c in colours:
            deg = ptr[c + 1] - ptr[c]
            k = corner[np.repeat(ptr[c] - np.concatenate([[0], np.cumsum(deg)[:-1]]), deg) + np.arange(deg.sum())]
            self.sets.append(tuple(torch.as_tensor(q, device=self.dev) for q in (c, np.repeat(np.arange(c.size), deg), k // 4, k % 4)))
        self.mu, self.lam = (self.t(np.concatenate([m[k] for m in meshes])) for k in ("mu", "lam"))
        self.x, self.v = self.t(X), self.t(np.concatenate([m["v"] for m in meshes]))
        self.kD, self.rho = case.get("kD") or 0.0, case.get("rho") or 0.0
        self.strategy = case.get("strategy", 2 if case["kind"] == "rollout" else 4)

    def t(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)

    def solve(self, x, xt, target, h, s):
        """The Newton step of the vertices of one colour set."""
        c, owner, e, il = s
        F = torch.einsum("eai,eaj->eij", x[self.T[e]], self.grads[e])
        w = self.grads[e, il]
        J1 = torch.linalg.cross(F[:, :, 1], F[:, :, 2])
        J2 = torch.linalg.cross(F[:, :, 2], F[:, :, 0])
        J3 = torch.linalg.cross(F[:, :, 0], F[:, :, 1])
        J = (F[:, :, 0] * J1).sum(1)
        p = w[:, :1] * J1 + w[:, 1:2] * J2 + w[:, 2:] * J3
        vm, vl = self.vol[e] * self.mu[e], self.vol[e] * self.lam[e]
        alpha = 1.0 + self.mu[e] / self.lam[e]
        ge = vm[:, None] * torch.einsum("eij,ej->ei", F, w) + (vl * (J - alpha))[:, None] * p
        He = (vm * (w * w).sum(1))[:, None, None] * torch.eye(3, dtype=torch.float64, device=self.dev) + vl[:, None, None] * p[:, :, None] * p[:, None, :]
        g = torch.zeros((c.numel(), 3), dtype=torch.float64, device=self.dev).index_add(0, owner, ge)
        H = torch.zeros((c.numel(), 3, 3), dtype=torch.float64, device=self.dev).index_add(0, owner, He)
        if self.kD:
            D = self.kD / h
            g = g + D * torch.einsum("eij,ej->ei", H, x[c] - xt[c])
            H = H * (1.0 + D)
        K = (self.m[c] / h**2)[:, None]
        g = g + K * (x[c] - target[c])
        H = H + K[:, :, None] * torch.eye(3, dtype=torch.float64, device=self.dev)
        # The symmetric 3 x 3 solve by the adjugate.
        adj = torch.stack([torch.linalg.cross(H[:, 1], H[:, 2]), torch.linalg.cross(H[:, 2], H[:, 0]),
                           torch.linalg.cross(H[:, 0], H[:, 1])], dim=1)
        det = (H[:, 0] * adj[:, 0]).sum(1)
        return x[c] - torch.einsum("eij,ej->ei", adj, g) / det[:, None]

    def step(self, x, v, dt, iterations, substeps):
        h = dt / substeps
        for _ in range(substeps):
            xt = x
            target = xt + h * v + h * h * self.a
            if self.strategy == 2:
                x = target
            else:
                vn = v.norm(dim=1, keepdim=True) + np.finfo(np.float32).tiny
                an = (self.a * self.a).sum(1, keepdim=True)
                f = ((v / vn) * self.a).sum(1, keepdim=True).abs() / torch.where(an > 0, an, torch.ones_like(an))
                x = xt + h * v + h * h * f.clamp(max=1.0) * self.a
            omega, back = 0.0, [x, x]
            for k in range(iterations):
                for s in self.sets:
                    x = x.index_put((s[0],), self.solve(x, xt, target, h, s))
                if self.rho:
                    omega = 1.0 if k == 0 else 2.0 / (2.0 - self.rho**2) if k == 1 else 1.0 - self.rho**2 * omega
                    if k > 1:
                        x = omega * (x - back[0]) + back[0]
                    back = [back[1], x]
            v = (x - xt) / h
        return x, v


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("step", "batch", "rollout"):
        return None
    meshes = _meshes(case, seed)
    # FP64 sweeps of the largest meshes, and the graph of a long rollout, take minutes.
    nv, nt = _counts(case)
    sweeps = 8.0 * case["iterations"] * case.get("substeps", 1) * case.get("steps", 1)
    if nt * sweeps > 8e8 or (kind == "rollout" and sweeps > 500):
        return None
    E = _Exact(meshes, case)
    if kind != "rollout":
        with torch.no_grad():
            x, v = E.step(E.x, E.v, DT, case["iterations"], case.get("substeps", 1))
        return dict(x=x, v=v)
    leaves = [a.requires_grad_() for a in (E.x, E.v)]
    x, v = leaves
    for _ in range(case["steps"]):
        x, v = E.step(x, v, DT, case["iterations"], 1)
    ((x - E.X) ** 2).sum().backward()
    return dict(x=x.detach(), v=v.detach(), dx0=leaves[0].grad, dv0=leaves[1].grad)
