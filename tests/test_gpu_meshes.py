"""Steps of meshes that are not hex grids, against the FP64 oracle: a Delaunay mesh whose stiffness varies from
tet to tet, tets that meet in ways a manifold mesh does not have, and a vertex with more neighbours than the
slots of a pair of incidences can name (every incidence is then a pair by itself, gathered from the tets).  The
cluster step, the launches per colour and the recorded step give the same positions bit for bit."""

import numpy as np
import pytest

import oracle_lib as O
from physicsbasedanimationtoolkit_gb300 import _capi, meshgen, pbat

spatial = pytest.importorskip("scipy.spatial")
pytestmark = pytest.mark.gpu

TOL = 1e-4  # of the bounding-box diagonal


def oriented(X, T):
    """The tets with positive volume, corners swapped where needed; flat ones left out."""
    T = np.array(T)
    e = X[T[:, 1:]] - X[T[:, :1]]
    d = np.linalg.det(e)
    T[d < 0] = T[d < 0][:, [0, 2, 1, 3]]
    h = np.abs(e).max(axis=(1, 2))
    return T[np.abs(d) > 1e-2 * h**3]


def delaunay(seed):
    """Jittered points of a box, all tets of their Delaunay mesh but the flat ones."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(np.arange(9), np.arange(6), np.arange(6), indexing="ij"), -1).reshape(-1, 3)
    X = (g + rng.uniform(-0.25, 0.25, g.shape)) / 6.0
    T = oriented(X, spatial.Delaunay(X).simplices)
    # A random rotation of each tet's corners (an even permutation keeps the volume's sign).
    even = np.array([[0, 1, 2, 3], [0, 2, 3, 1], [0, 3, 1, 2], [1, 0, 3, 2], [1, 3, 2, 0], [2, 3, 0, 1], [3, 2, 1, 0]])
    T = np.take_along_axis(T, even[rng.integers(0, len(even), T.shape[0])], axis=1)
    return X, T, np.nonzero(X[:, 0] < 0.2)[0]


def non_manifold(seed):
    """Two blocks that share one edge, a third that shares one vertex with them, and tets three to a face."""
    X, T = meshgen.hex_grid(3, 2, 2, hi=(1.5, 1.0, 1.0))
    n = X.shape[0]
    hi = X[:, 0].max()
    edge = np.nonzero((X[:, 0] == hi) & (X[:, 1] == 1.0))[0][:2]
    blocks, tets = [X], [T]
    for k, shared in enumerate((edge, edge[:1])):
        Y = X + np.array([hi, 1.0, 0.0]) * (1 if k == 0 else -1) + (0 if k == 0 else np.array([2 * hi, 2.0, 0.7]))
        ids = n * (k + 1) + np.arange(n)
        # Move the second mesh so that its corner lies on the shared vertices, then merge those.
        for s in shared:
            near = np.argmin(np.linalg.norm(Y - X[s], axis=1))
            ids[near], Y[near] = s, X[s]
        blocks.append(Y)
        tets.append(ids[T])
    X, T = np.concatenate(blocks), np.concatenate(tets)
    tip = X[:n].mean(0) + np.array([[0.1, 0.9, 1.3], [0.3, 1.1, 1.6]])
    top = T[np.argmax(X[T].mean(1)[:, 2])]
    face = [v for v in top if v != top[np.argmin(X[top][:, 2])]]
    extra = [face + [X.shape[0]], face + [X.shape[0] + 1]]
    X, T = np.concatenate([X, tip]), np.concatenate([T, extra])
    used, T = np.unique(oriented(X, T), return_inverse=True)
    X, T = X[used], T.reshape(-1, 4)
    return X, T, np.nonzero(X[:, 0] == 0.0)[0]


def hub(seed):
    """A ball of tets that all meet in its centre: 320 neighbours."""
    n = 320
    k = np.arange(n) + 0.5
    phi, z = np.pi * (1 + 5**0.5) * k, 1 - 2 * k / n
    P = np.stack([np.cos(phi) * np.sqrt(1 - z * z), np.sin(phi) * np.sqrt(1 - z * z), z], 1)
    hull = spatial.ConvexHull(P).simplices
    X = np.concatenate([P, np.zeros((1, 3))])
    e = X[hull]
    T = np.concatenate([np.full((hull.shape[0], 1), n), hull], 1)
    d = np.linalg.det(e)
    T[d < 0] = T[d < 0][:, [0, 2, 1, 3]]
    return X, T, np.nonzero(z < -0.9)[0]


MESHES = dict(delaunay=delaunay, non_manifold=non_manifold, hub=hub)


def problem(name, seed=0, **kw):
    X, T, dbc = MESHES[name](seed)
    rng = np.random.default_rng(seed + 1)
    E = 3e5 * np.exp(rng.uniform(-1.5, 1.5, T.shape[0]))
    mu, lam = meshgen.lame(E, rng.uniform(0.2, 0.45, T.shape[0]))
    rho = np.full(T.shape[0], 1000.0)
    v = rng.uniform(-0.2, 0.2, X.shape)
    d = (pbat.sim.vbd.Data().with_volume_mesh(X.T, T.T).with_material(rho, mu, lam).with_dirichlet_vertices(dbc)
         .with_velocity(v.T).with_initialization_strategy(kw.get("strategy", 2)))
    if kw.get("rho"):
        d = d.with_chebyshev_acceleration(kw["rho"])
    if kw.get("kD"):
        d = d.with_rayleigh_damping(kw["kD"])
    oracle = O.OracleVbd(X, T, rho, mu, lam, dbc, v=v, strategy=kw.get("strategy", 2), semantics=1,
                         rho_chebyshev=kw.get("rho"), kD=kw.get("kD", 0.0))
    return d.construct(), oracle, X, T


@pytest.mark.parametrize("kw", [dict(), dict(rho=0.8, kD=1e-3, strategy=3)])
@pytest.mark.parametrize("name", list(MESHES))
def test_irregular_mesh_matches_oracle(name, kw):
    d, R, X, T = problem(name, **kw)
    A, B, C = (pbat.gpu.vbd.Integrator(d) for _ in range(3))
    _capi.check(_capi.lib().pbgb_vbd_set_persistent(B.handle, 0), B.handle)
    C.adjoint_reserve(2, 10)
    staged = A.staged_sweep[0]
    assert staged == (name != "hub")
    if not staged:
        assert max(np.unique(T[(T == i).any(1)]).size - 1 for i in range(X.shape[0])) > 256
    for _ in range(4):
        for I in (A, B):
            I.step(1 / 60, 10, 2)
        C.step_record(1 / 60, 10, 2, 0)
    assert A.launches_per_step(10, 2) == 1 if staged else A.launches_per_step(10, 2) > 1
    np.testing.assert_array_equal(A.x, B.x)
    np.testing.assert_array_equal(A.x, C.x)
    R.step(1 / 60, 10, 2, 4)
    diag = np.linalg.norm(X.max(0) - X.min(0))
    assert np.abs(A.x.T - R.x).max() / diag <= TOL
    assert np.abs(R.x - X).max() / diag > 1e-3


@pytest.mark.parametrize("lanes", [1, 4, 32])
def test_irregular_meshes_in_a_batch(lanes):
    """In clusters, by tickets and in launches per colour; each mesh as by itself."""
    names = ("delaunay", "non_manifold", "delaunay")
    parts = [problem(name, seed) for seed, name in enumerate(names)]
    datas = [p[0] for p in parts]
    A, B, T = (pbat.gpu.vbd.BatchedIntegrator(datas) for _ in range(3))
    B.persistent = False
    _capi.check(_capi.lib().pbgb_debug_batched_wait(T.handle, 2_000_000_000, 2**30), T.handle)
    singles = [pbat.gpu.vbd.Integrator(d) for d in datas]
    for I in (A, B, T, *singles):
        I.lanes_per_vertex = lanes
        for _ in range(2):
            I.step(1 / 60, 8, 1)
    for I in (B, T):
        np.testing.assert_array_equal(A.x, I.x)
    off = A.vertex_offsets
    for b, s in enumerate(singles):
        np.testing.assert_array_equal(A.x[:, off[b]: off[b + 1]], s.x)


@pytest.mark.parametrize("name", list(MESHES))
def test_reversed_steps_of_irregular_meshes(name):
    """The reversed chain against the sweeps with atomics: the same FP32 terms summed in other orders."""
    torch = pytest.importorskip("torch")
    d = problem(name, rho=0.8, kD=1e-3)[0]
    out = []
    for on in (1, 0):
        I = pbat.gpu.vbd.Integrator(d)
        _capi.check(_capi.lib().pbgb_vbd_set_persistent(I.handle, on), I.handle)
        x0, v0 = (torch.tensor(np.ascontiguousarray(a.T), dtype=torch.float32, device="cuda", requires_grad=True) for a in (d.X, d.v))
        mu, lam = (torch.tensor(m, requires_grad=True) for m in d.lame)
        x, v = pbat.gpu.vbd.rollout(I, mu, lam, x0, v0, dt=1 / 60, iterations=6, steps=2, substeps=2)
        ((x ** 2).sum() + (v ** 2).sum()).backward()
        out.append([g.grad.cpu().numpy() for g in (x0, v0, mu, lam)])
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)
