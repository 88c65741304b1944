"""The cluster step (one launch per step, a mesh's parts in the blocks of a thread-block cluster) against
launches per colour: the per-vertex arithmetic, its order and the lanes are the same, so positions and
velocities must be equal bit for bit, whatever the number of blocks, the ring of tiles or the rounds of a
colour; and a recorded rollout must tape the same iterates."""

import time

import numpy as np
import pytest

from physicsbasedanimationtoolkit_gb300 import _capi, meshgen, pbat

pytestmark = pytest.mark.gpu


def data_of(nx, ny, nz, rho=None, kD=0.0, strategy=4, seed=0):
    X, T = meshgen.hex_grid(nx, ny, nz, hi=(nx / nz, ny / nz, 1.0))
    dbc = meshgen.face_vertices(X, 0, 0.0)
    X = meshgen.jitter(X, 0.02 / nz, seed)
    mu, lam = meshgen.lame(np.full(T.shape[0], 1e6), np.full(T.shape[0], 0.45))
    v = np.random.default_rng(seed).uniform(-0.5, 0.5, X.shape)
    d = (pbat.sim.vbd.Data().with_volume_mesh(X.T, T.T).with_material(np.full(T.shape[0], 1000.0), mu, lam)
         .with_dirichlet_vertices(dbc).with_velocity(v.T).with_initialization_strategy(strategy))
    if rho is not None:
        d = d.with_chebyshev_acceleration(rho)
    if kD:
        d = d.with_rayleigh_damping(kD)
    return d.construct()


def set_persistent(I, on):
    _capi.check(_capi.lib().pbgb_vbd_set_persistent(I.handle, int(on)), I.handle)


# Sizes: one hex (4 free vertices), 1 to 16 blocks, parts of uneven size, parts whose tiles do not all
# fit the ring (20^3), and the smallest mesh past the limit.  Lanes 1 and 32 give several rounds of
# groups per colour and tiles shared by many warps.
@pytest.mark.parametrize("shape,lanes", [((1, 1, 1), 0), ((3, 2, 2), 32), ((5, 4, 4), 0), ((7, 5, 4), 8), ((9, 9, 9), 4),
                                         ((31, 7, 6), 0), ((13, 11, 10), 32), ((16, 16, 16), 1), ((20, 20, 20), 0),
                                         ((20, 20, 20), 2), ((20, 20, 22), 0)])
@pytest.mark.parametrize("mode", ["plain", "chebyshev_damped_substeps"])
def test_cluster_step_equals_colour_launches(shape, lanes, mode):
    kw, sub = ({}, 1) if mode == "plain" else (dict(rho=0.85, kD=1e-3, strategy=3), 2)
    d = data_of(*shape, **kw)
    A, B = pbat.gpu.vbd.Integrator(d), pbat.gpu.vbd.Integrator(d)
    for I in (A, B):
        I.lanes_per_vertex = lanes
    set_persistent(B, False)
    for _ in range(3):
        A.step(1 / 60, 6, sub)
        B.step(1 / 60, 6, sub)
    assert A.launches_per_step(6, sub) == (1 if A.n_free <= 9000 else B.launches_per_step(6, sub))
    assert B.launches_per_step(6, sub) > 1
    np.testing.assert_array_equal(A.x, B.x)
    np.testing.assert_array_equal(A.v, B.v)


@pytest.mark.parametrize("n_meshes,nmin,nmax", [(1, 3, 3), (3, 1, 12), (9, 2, 9), (40, 2, 5)])
def test_cluster_batch_equals_colour_launches(n_meshes, nmin, nmax):
    datas = [data_of(n, n, n, rho=0.8, seed=n) for n in np.linspace(nmin, nmax, n_meshes).astype(int)]
    A, B = pbat.gpu.vbd.BatchedIntegrator(datas), pbat.gpu.vbd.BatchedIntegrator(datas)
    B.persistent = False
    for _ in range(2):
        A.step(1 / 60, 5, 2)
        B.step(1 / 60, 5, 2)
    assert A.launches_per_step(5, 2) == 1
    np.testing.assert_array_equal(A.x, B.x)
    np.testing.assert_array_equal(A.v, B.v)


@pytest.mark.parametrize("rho", [None, 0.85])
@pytest.mark.parametrize("shape", [(2, 2, 2), (12, 5, 4)])
def test_recorded_cluster_rollout_equals_colour_launches(shape, rho):
    torch = pytest.importorskip("torch")
    d = data_of(*shape, rho=rho, strategy=2)
    out = []
    for on in (True, False):
        I = pbat.gpu.vbd.Integrator(d)
        set_persistent(I, on)
        x0 = torch.tensor(np.ascontiguousarray(d.X.T), dtype=torch.float32, device="cuda", requires_grad=True)
        v0 = torch.tensor(np.ascontiguousarray(d.v.T), dtype=torch.float32, device="cuda", requires_grad=True)
        mu, lam = torch.tensor(d.lame[0]), torch.tensor(d.lame[1])
        x, v = pbat.gpu.vbd.rollout(I, mu, lam, x0, v0, dt=1 / 60, iterations=6, steps=3, substeps=2, checkpoint_every=2)
        ((x ** 2).sum() + (v ** 2).sum()).backward()
        out.append((x.detach().cpu().numpy(), v.detach().cpu().numpy(), x0.grad.cpu().numpy(), v0.grad.cpu().numpy()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    # The same tape; the reversed sweeps add to neighbours' adjoints with FP32 atomics in any order.
    for a, b in zip(out[0][2:], out[1][2:]):
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)


# The reversed chain of small meshes (blocks, chain, material sensitivities) against the sweeps with
# atomics: one hex, a turn that fills its groups exactly or not, colours up to the limit and past it (both
# sides take the sweeps then), iterations past one workspace, and the two sums it does not share with plain
# iterations (damping, Chebyshev carries).  Both sum the same FP32 terms in other orders; two runs of the
# chain give the same bits.
@pytest.mark.parametrize("rho,kD", [(None, 0.0), (0.85, 0.0), (None, 1e-3), (0.8, 1e-3)])
@pytest.mark.parametrize("shape,iterations", [((1, 1, 1), 3), ((4, 3, 2), 1), ((7, 3, 3), 7), ((10, 6, 6), 4), ((10, 6, 6), 70), ((15, 5, 5), 4)])
def test_reversed_chain_equals_sweeps_with_atomics(shape, iterations, rho, kD):
    torch = pytest.importorskip("torch")
    d = data_of(*shape, rho=rho, kD=kD, strategy=2)
    weight = torch.tensor(np.random.default_rng(3).uniform(-1, 1, (d.X.shape[1], 3)), dtype=torch.float32, device="cuda")
    out = []
    for on in (True, True, False):
        I = pbat.gpu.vbd.Integrator(d)
        set_persistent(I, on)
        x0 = torch.tensor(np.ascontiguousarray(d.X.T), dtype=torch.float32, device="cuda", requires_grad=True)
        v0 = torch.tensor(np.ascontiguousarray(d.v.T), dtype=torch.float32, device="cuda", requires_grad=True)
        mu, lam = (torch.tensor(m, requires_grad=True) for m in d.lame)
        x, v = pbat.gpu.vbd.rollout(I, mu, lam, x0, v0, dt=1 / 60, iterations=iterations, steps=2, substeps=2)
        ((weight * x).sum() + (v ** 2).sum()).backward()
        out.append([g.grad.cpu().numpy() for g in (x0, v0, mu, lam)])
    for a, b, c in zip(*out):
        np.testing.assert_array_equal(a, b) if shape != (15, 5, 5) else None
        assert np.linalg.norm(a - c) <= 1e-4 * np.linalg.norm(c)


# A tile that never arrives: resident and streamed tiles, one block and several (the others then wait for
# positions that do not come), the first tile and a later one, of a later iteration where tiles are streamed,
# and a batch.  The step ends with PBGB_ERR_TIMEOUT soon after the limit, and after the hook is cleared the
# same step from the same state is that of an integrator that never timed out.
@pytest.mark.parametrize("shapes,lanes,tile", [([(2, 2, 2)], 0, 0), ([(9, 9, 9)], 4, 0), ([(9, 9, 9)], 0, 3),
                                               ([(20, 20, 20)], 2, 0), ([(20, 20, 20)], 2, 40), ([(20, 20, 20)], 0, 25),
                                               ([(2, 2, 2), (5, 5, 5), (7, 7, 7)], 0, 1)])
@pytest.mark.parametrize("rho,substeps", [(None, 1), (0.85, 2)])
def test_a_cluster_wait_that_runs_out_reports_a_timeout_and_the_context_survives(shapes, lanes, tile, rho, substeps):
    datas = [data_of(*s, rho=rho, strategy=2) for s in shapes]
    A, B = (pbat.gpu.vbd.BatchedIntegrator(datas) if len(datas) > 1 else pbat.gpu.vbd.Integrator(datas[0]) for _ in range(2))
    for I in (A, B):
        I.lanes_per_vertex = lanes
    L = _capi.lib()
    x0, v0 = A.x, A.v
    for _ in range(2):
        _capi.check(L.pbgb_debug_cluster_wait(A.handle, 5_000_000, tile), A.handle)
        A.step(1 / 60, 8, substeps)
        start = time.perf_counter()
        with pytest.raises(_capi.PbgbError) as err:
            A.synchronize()
        assert err.value.code == 7
        assert time.perf_counter() - start < 1.0
        assert A.launches_per_step(8, substeps) == 1
        _capi.check(L.pbgb_debug_cluster_wait(A.handle, 2_000_000_000, -1), A.handle)
        A.x, A.v = x0, v0
        A.step(1 / 60, 8, substeps)
        A.synchronize()
        if _ == 0:
            B.step(1 / 60, 8, substeps)
        np.testing.assert_array_equal(A.x, B.x)
        np.testing.assert_array_equal(A.v, B.v)


def test_a_recorded_cluster_step_that_times_out():
    d = data_of(9, 9, 9, rho=0.85, strategy=2)
    A, B = pbat.gpu.vbd.Integrator(d), pbat.gpu.vbd.Integrator(d)
    L = _capi.lib()
    x0, v0 = A.x, A.v
    for I in (A, B):
        I.adjoint_reserve(2, 6)
    _capi.check(L.pbgb_debug_cluster_wait(A.handle, 5_000_000, 2), A.handle)
    A.step_record(1 / 60, 6, 2, 0)
    with pytest.raises(_capi.PbgbError) as err:
        A.synchronize()
    assert err.value.code == 7
    _capi.check(L.pbgb_debug_cluster_wait(A.handle, 2_000_000_000, -1), A.handle)
    A.x, A.v = x0, v0
    for I in (A, B):
        I.step_record(1 / 60, 6, 2, 0)
    np.testing.assert_array_equal(A.x, B.x)


def test_the_cluster_hook_rejects_out_of_range_limits():
    I = pbat.gpu.vbd.Integrator(data_of(2, 2, 2))
    L = _capi.lib()
    for ns, tile in ((10, -1), (5_000_000_000, -1), (1_000_000, -2)):
        assert L.pbgb_debug_cluster_wait(I.handle, ns, tile) == 1


@pytest.mark.parametrize("shape", [(4, 3, 3), (20, 20, 20)])
def test_damping_switched_on_and_off(shape):
    """The step's shared memory holds more with damping: a launch made without is not used with it."""
    d = data_of(*shape, rho=0.85)
    A, B = pbat.gpu.vbd.Integrator(d), pbat.gpu.vbd.Integrator(d)
    set_persistent(B, False)
    for kD in (0.0, 1e-3, 0.0, 1e-2):
        for I in (A, B):
            I.kD = kD
            I.step(1 / 60, 5, 1)
        np.testing.assert_array_equal(A.x, B.x)
        np.testing.assert_array_equal(A.v, B.v)
    assert A.launches_per_step(5, 1) == 1


def test_chebyshev_weights_of_many_iterations():
    """The weights of a longer step are on the device before its kernel reads them (80 KB: more than a copy from
    pageable memory stages at once): the first such step equals a later one."""
    d = data_of(2, 2, 2, rho=0.9, strategy=2)
    I = pbat.gpu.vbd.Integrator(d)
    x0, v0 = I.x, I.v
    out = []
    for _ in range(2):
        I.x, I.v = x0, v0
        I.step(1 / 60, 20000, 1)
        out.append((I.x, I.v))
    np.testing.assert_array_equal(out[0], out[1])


def test_a_step_whose_weights_find_no_room():
    """The call says so; the next one makes the weights again, also a shorter step that the lost ones covered."""
    d = data_of(3, 3, 3, rho=0.9, strategy=2)
    A, B = pbat.gpu.vbd.Integrator(d), pbat.gpu.vbd.Integrator(d)
    L = _capi.lib()
    for I in (A, B):
        I.step(1 / 60, 10, 1)
    _capi.check(L.pbgb_debug_fail_allocation(0, None))
    with pytest.raises(_capi.PbgbError):
        A.step(1 / 60, 20, 1)
    for n in (5, 30):
        for I in (A, B):
            I.step(1 / 60, n, 1)
        np.testing.assert_array_equal(A.x, B.x)
