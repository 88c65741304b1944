"""GPU LBVH against the oracle: Morton codes, sort order, topology and internal boxes bit-exact;
overlap pair sets equal to brute force."""

import json
import pathlib
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import oracle_lib as O
from physicsbasedanimationtoolkit_gb300 import _capi, meshgen, pbat

pytestmark = pytest.mark.gpu

GOLD = pathlib.Path(__file__).resolve().parent / "golden"


def gpu_build(lo, hi, wmin, wmax):
    bvh = pbat.gpu.geometry.Bvh(lo.shape[0], 0)
    bvh.build(lo.T, hi.T, wmin, wmax)
    return bvh, bvh._topology()


def assert_same(g, o):
    np.testing.assert_array_equal(g["codes"], o["codes"])
    np.testing.assert_array_equal(g["inds"], o["inds"])
    np.testing.assert_array_equal(g["child"], o["child"])
    np.testing.assert_array_equal(g["parent"], o["parent"])
    np.testing.assert_array_equal(g["rightmost"], o["rightmost"])
    np.testing.assert_array_equal(g["ilo"], o["ilo"])
    np.testing.assert_array_equal(g["ihi"], o["ihi"])


def test_cube_topology_known_answer_on_device():
    kat = json.loads((GOLD / "kat.json").read_text())["bvh_cube5"]
    P, T, _, _ = meshgen.cube5()
    X = P.T.astype(np.float32)
    pts = X[T.T]
    lo, hi = pts.min(axis=1), pts.max(axis=1)
    _, g = gpu_build(lo, hi, X.min(axis=0), X.max(axis=0))
    np.testing.assert_array_equal(g["child"], np.array(kat["child"]))
    np.testing.assert_array_equal(g["parent"], np.array(kat["parent"]))
    np.testing.assert_array_equal(g["rightmost"], np.array(kat["rightmost"]))


def test_morton_codes_match_reference_fixture_on_device():
    g = np.load(GOLD / "morton.npz")
    _, t = gpu_build(g["lo"], g["hi"], g["wmin"], g["wmax"])
    expected = np.sort(g["codes"], kind="stable")
    np.testing.assert_array_equal(t["codes"], expected)
    np.testing.assert_array_equal(t["inds"], np.argsort(g["codes"], kind="stable"))


def scene_boxes(swept):
    w = meshgen.contact_scene_workload()
    X = w["X"].astype(np.float32)
    Xn = None
    if swept:
        Xn = (X + np.random.default_rng(1).uniform(-0.01, 0.01, X.shape) + np.array([0, 0, -0.02])).astype(np.float32)
    lo, hi = meshgen.triangle_boxes(X, w["F"], Xn)
    lo, hi = lo.astype(np.float32), hi.astype(np.float32)
    allp = X if Xn is None else np.vstack([X, Xn])
    return w, lo, hi, allp.min(axis=0), allp.max(axis=0)


@pytest.mark.parametrize("swept", [False, True])
def test_scene_triangle_bvh_bit_exact(swept):
    """66,560 surface triangles of the 16-cube contact scene."""
    w, lo, hi, wmin, wmax = scene_boxes(swept)
    assert lo.shape[0] == 66560
    _, g = gpu_build(lo, hi, wmin, wmax)
    o = O.bvh_build(lo, hi, wmin, wmax)
    assert_same(g, o)


@pytest.mark.parametrize("n", [2, 3, 1000, 1024, 1025, 2049, 200_000, 1_100_000])
def test_random_boxes_with_duplicate_codes(n):
    rng = np.random.default_rng(n)
    lo = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    hi = (lo + rng.uniform(0, 0.01, (n, 3))).astype(np.float32)
    lo[: n // 3] = lo[n // 3: 2 * (n // 3)]
    hi[: n // 3] = hi[n // 3: 2 * (n // 3)]
    _, g = gpu_build(lo, hi, [0, 0, 0], [1.01, 1.01, 1.01])
    assert_same(g, O.bvh_build(lo, hi, [0, 0, 0], [1.01, 1.01, 1.01]))


# Codes and sort of one block: rounds of a warp partly filled, the tile full and one box past it; boxes
# that share one code or a few (the sort must keep their order).
@pytest.mark.parametrize("n", [31, 256, 257, 4095, 4096, 4097])
@pytest.mark.parametrize("codes", [1, 5, 0])
def test_sort_of_one_tile(n, codes):
    rng = np.random.default_rng(n)
    lo = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    if codes:
        lo = lo[rng.integers(0, codes, n)]
    hi = (lo + np.float32(0.01)).astype(np.float32)
    _, g = gpu_build(lo, hi, [0, 0, 0], [1.01, 1.01, 1.01])
    assert_same(g, O.bvh_build(lo, hi, [0, 0, 0], [1.01, 1.01, 1.01]))


def test_overlap_pairs_equal_brute_force():
    w, lo, hi, wmin, wmax = scene_boxes(True)
    X = w["X"].astype(np.float32)
    rng = np.random.default_rng(7)
    V = w["V"][rng.choice(w["V"].size, 4000, replace=False)]
    Xn = X + np.array([0, 0, -0.03], np.float32)
    qlo = np.minimum(X[V], Xn[V])
    qhi = np.maximum(X[V], Xn[V])
    bvh, _ = gpu_build(lo, hi, wmin, wmax)
    got = bvh.overlaps(qlo.T, qhi.T)
    exp = O.overlaps(lo, hi, qlo, qhi)
    assert exp.shape[0] > 1000
    assert {tuple(p) for p in got.T} == {tuple(p) for p in exp}
    assert got.shape[1] == exp.shape[0]


def test_refit_matches_oracle_boxes_for_same_topology():
    w, lo, hi, wmin, wmax = scene_boxes(False)
    bvh, g0 = gpu_build(lo, hi, wmin, wmax)
    X = w["X"].astype(np.float32) + np.random.default_rng(3).uniform(-0.02, 0.02, w["X"].shape).astype(np.float32)
    lo2, hi2 = meshgen.triangle_boxes(X, w["F"])
    lo2, hi2 = lo2.astype(np.float32), hi2.astype(np.float32)
    bvh.refit(lo2.T, hi2.T)
    g = bvh._topology()
    np.testing.assert_array_equal(g["child"], g0["child"])
    ilo, ihi = O.bvh_boxes(g["child"], g["inds"], lo2, hi2)
    np.testing.assert_array_equal(g["ilo"], ilo)
    np.testing.assert_array_equal(g["ihi"], ihi)


def test_build_from_device_boxes_equals_host_build():
    """pbgb_bvh_build_device (boxes already on the device) gives the same codes, order, topology
    and boxes as the host-buffer build, and both equal the oracle."""
    import ctypes as C

    import torch

    from physicsbasedanimationtoolkit_gb300 import _capi

    rng = np.random.default_rng(21)
    n = 20000
    c = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    e = rng.uniform(0, 0.01, (n, 3)).astype(np.float32)
    lo, hi = (c - e).astype(np.float32), (c + e).astype(np.float32)
    wmin, wmax = np.zeros(3, np.float32), np.ones(3, np.float32)
    bvh, host = gpu_build(lo, hi, wmin, wmax)
    lo4 = torch.zeros((n, 4), device="cuda")
    hi4 = torch.zeros((n, 4), device="cuda")
    lo4[:, :3] = torch.from_numpy(lo).cuda()
    hi4[:, :3] = torch.from_numpy(hi).cuda()
    torch.cuda.synchronize()
    L = _capi.lib()
    _capi.check_bvh(L.pbgb_bvh_build_device(bvh._h, n, C.c_void_p(lo4.data_ptr()), C.c_void_p(hi4.data_ptr()),
                                            wmin.ctypes.data, wmax.ctypes.data), bvh._h)
    dev = bvh._topology()
    assert_same(dev, host)
    assert_same(dev, O.bvh_build(lo, hi, wmin, wmax))


# ---------------------------------------------------------------------------------------------
# The reference binding's remaining queries (bindings/pypbat/gpu/geometry/Bvh.cpp, Aabb.cpp).

def _brute_self_overlaps(lo, hi, sets=None):
    """Unordered pairs {i, j}, i != j, of closed boxes that overlap (numpy, exact comparisons)."""
    ov = np.all((lo[:, None, :] <= hi[None, :, :]) & (lo[None, :, :] <= hi[:, None, :]), axis=2)
    i, j = np.nonzero(np.triu(ov, 1))
    keep = np.ones(i.size, bool) if sets is None else sets[i] != sets[j]
    return {frozenset((a, b)) for a, b in zip(i[keep].tolist(), j[keep].tolist())}


def test_detect_overlaps_between_sets_reference_case():
    """The reference's doctest (gpu/geometry/Bvh.cu:336-404): three edges (set 0) and one
    triangle (set 1); the triangle overlaps edges 1 and 0, each pair reported once."""
    V = np.array([[0, 1, 2, 3, 0, 2, 0], [0, 0.1, 0.2, 0.3, 0, 0.1, 0], [0, 10, 20, 30, 0, 10, 0]], np.float32)
    E1 = np.array([[1, 0, 2], [2, 1, 3]])
    F2 = np.array([[4], [5], [6]])
    edges, tris = pbat.gpu.geometry.Aabb(3, 3), pbat.gpu.geometry.Aabb(3, 1)
    edges.construct(V, E1)
    tris.construct(V, F2)
    L = np.hstack([edges.min, tris.min])
    U = np.hstack([edges.max, tris.max])
    aabbs = pbat.gpu.geometry.Aabb(3, 4)
    aabbs.construct(L, U)
    sets = np.array([0, 0, 0, 1], np.int32)
    bvh = pbat.gpu.geometry.Bvh(4, 4)
    bvh.build(aabbs, L.min(axis=1), U.max(axis=1))
    O2 = bvh.detect_overlaps(aabbs, sets)
    assert O2.shape == (2, 2)
    assert {frozenset(c) for c in O2.T.tolist()} == {frozenset((3, 1)), frozenset((3, 0))}
    assert (bvh.visits == 2).all()


@pytest.mark.parametrize("n", [2, 3, 50, 2000])
def test_self_overlaps_equal_brute_force(n):
    rng = np.random.default_rng(n)
    c = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    r = rng.uniform(0.005, 0.05, (n, 3)).astype(np.float32)
    lo, hi = c - r, c + r
    lo[: n // 10] = lo[n // 10: 2 * (n // 10)]  # duplicated boxes (equal Morton codes)
    hi[: n // 10] = hi[n // 10: 2 * (n // 10)]
    bvh = pbat.gpu.geometry.Bvh(n, 16)
    bvh.build(lo.T, hi.T, lo.min(axis=0), hi.max(axis=0))
    O1 = bvh.detect_overlaps(lo.T, upper=hi.T)
    got = [frozenset(p) for p in O1.T.tolist()]
    assert len(got) == len(set(got))  # each pair once
    assert set(got) == _brute_self_overlaps(lo, hi)
    sets = rng.integers(0, 3, n).astype(np.int32)
    O2 = bvh.detect_overlaps(lo.T, sets, upper=hi.T)
    got2 = [frozenset(p) for p in O2.T.tolist()]
    assert len(got2) == len(set(got2))
    assert set(got2) == _brute_self_overlaps(lo, hi, sets)


def _np_point_triangle(p, a, b, c):
    """FP64 point-triangle distance by Voronoi regions (independent of the device code)."""
    ab, ac, ap = b - a, c - a, p - a
    d1, d2 = ab @ ap, ac @ ap
    if d1 <= 0 and d2 <= 0:
        return np.linalg.norm(p - a)
    bp = p - b
    d3, d4 = ab @ bp, ac @ bp
    if d3 >= 0 and d4 <= d3:
        return np.linalg.norm(p - b)
    vc = d1 * d4 - d3 * d2
    if vc <= 0 and d1 >= 0 and d3 <= 0:
        return np.linalg.norm(p - (a + d1 / (d1 - d3) * ab))
    cp = p - c
    d5, d6 = ab @ cp, ac @ cp
    if d6 >= 0 and d5 <= d6:
        return np.linalg.norm(p - c)
    vb = d5 * d2 - d1 * d6
    if vb <= 0 and d2 >= 0 and d6 <= 0:
        return np.linalg.norm(p - (a + d2 / (d2 - d6) * ac))
    va = d3 * d6 - d5 * d4
    if va <= 0 and (d4 - d3) >= 0 and (d5 - d6) >= 0:
        return np.linalg.norm(p - (b + (d4 - d3) / ((d4 - d3) + (d5 - d6)) * (c - b)))
    den = 1.0 / (va + vb + vc)
    return np.linalg.norm(p - (a + ab * vb * den + ac * vc * den))


def _np_point_tet(p, a, b, c, d):
    def outside(u, v, w):
        return (p - u) @ np.cross(v - u, w - u) > 0
    if not (outside(a, b, d) or outside(b, c, d) or outside(c, a, d) or outside(a, c, b)):
        return 0.0
    return min(_np_point_triangle(p, a, b, d), _np_point_triangle(p, b, c, d), _np_point_triangle(p, c, a, d),
               _np_point_triangle(p, a, c, b))


def test_point_triangle_nearest_neighbours_are_nearest():
    """Nearest surface triangle of a jittered cube to points inside, near and far from it: the
    triangle returned is at the FP64 brute-force minimum distance (to FP32 rounding)."""
    w = meshgen.unit_cube_workload(n=6, seed=4)
    X = w["X"].astype(np.float64)
    F = meshgen.boundary_faces(w["T"]).astype(np.int32)
    aabbs = pbat.gpu.geometry.Aabb(3, F.shape[0])
    aabbs.construct(X.T, F.T)
    lo, hi = aabbs.min, aabbs.max
    np.testing.assert_array_equal(lo, X[F].min(axis=1).T.astype(np.float32))
    np.testing.assert_array_equal(hi, X[F].max(axis=1).T.astype(np.float32))
    bvh = pbat.gpu.geometry.Bvh(F.shape[0], 0)
    bvh.build(aabbs, lo.min(axis=1) - 1, hi.max(axis=1) + 1)
    rng = np.random.default_rng(2)
    P = np.vstack([rng.uniform(-0.5, 1.5, (300, 3)), rng.uniform(0.1, 0.9, (100, 3))]).astype(np.float32)
    nn = bvh.point_triangle_nearest_neighbours(aabbs, P.T, X.T, F.T)
    X32 = X.astype(np.float32).astype(np.float64)
    for q, f in enumerate(nn):
        d = np.array([_np_point_triangle(P[q].astype(np.float64), *X32[F[j]]) for j in range(F.shape[0])])
        assert 0 <= f < F.shape[0]
        assert d[f] <= d.min() + 1e-5


def test_point_tetrahedron_nearest_neighbours_are_nearest():
    """Nearest tetrahedron of a jittered cube: points inside get a tetrahedron that contains them
    (distance 0), points outside one at the FP64 brute-force minimum distance."""
    w = meshgen.unit_cube_workload(n=4, seed=6)
    X = w["X"].astype(np.float32)
    T = w["T"].astype(np.int32)
    aabbs = pbat.gpu.geometry.Aabb(3, T.shape[0])
    aabbs.construct(X.T, T.T)
    bvh = pbat.gpu.geometry.Bvh(T.shape[0], 0)
    bvh.build(aabbs, aabbs.min.min(axis=1), aabbs.max.max(axis=1))
    rng = np.random.default_rng(3)
    P = np.vstack([rng.uniform(0.05, 0.95, (200, 3)), rng.uniform(-0.4, 1.4, (100, 3))]).astype(np.float32)
    nn = bvh.point_tetrahedron_nearest_neighbours(aabbs, P.T, X.T, T.T)
    X64 = X.astype(np.float64)
    for q, t in enumerate(nn):
        d = np.array([_np_point_tet(P[q].astype(np.float64), *X64[T[j]]) for j in range(T.shape[0])])
        assert 0 <= t < T.shape[0]
        assert d[t] <= d.min() + 1e-5


@pytest.mark.parametrize("n,scale,offset", [(1, 1.0, 0.0), (2, 0.5, 3.0), (9, 1.0, 0.0), (16, 4.0, -64.0), (33, 0.25, 128.0)])
@pytest.mark.parametrize("height", [0.0, 0.5, 1024.0])
def test_nearest_triangle_among_exact_ties(n, scale, offset, height):
    """Queries over the vertices, edge middles and face interiors of a flat sheet whose coordinates are
    dyadic, so that every squared distance is rounded once and ties are many: the pick is the last of the first 8
    nearest triangles in decreasing leaf order, whatever the query passes over on its way."""
    i, j = (a.ravel() for a in np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij"))
    P = np.stack([i * scale + offset, j * scale + offset, 0.0 * i], 1).astype(np.float32)
    a, b = (c.ravel() for c in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    v = a * (n + 1) + b
    F = np.concatenate([np.stack([v, v + n + 1, v + n + 2], 1), np.stack([v, v + n + 2, v + 1], 1)])
    Q = np.concatenate([P, P + [scale / 2, 0, 0], P + [scale / 2, scale / 2, 0], P + [scale / 2, scale / 4, 0],
                        P - [4 * scale, 0, 0]]).astype(np.float32)
    Q[:, 2] = height
    bvh = pbat.gpu.geometry.Bvh(F.shape[0])
    boxes = pbat.gpu.geometry.Aabb()
    boxes.construct(P.T, F.T)
    bvh.build(boxes, P.min(0) - 1, P.max(0) + 1)
    nn = bvh.point_triangle_nearest_neighbours(boxes, Q.T, P.T, F.T)
    # Squared distances to the nearest point of a right triangle of the sheet, exact in FP64 and then
    # rounded to FP32 with the height's square (which hides small differences far above the sheet).
    A = P[F].astype(np.float64)
    q = Q[:, None, :2].astype(np.float64)
    lo, hi = A[:, :, :2].min(1), A[:, :, :2].max(1)
    c = np.clip(q, lo, hi)
    u = (c - lo) / (hi - lo)
    lower = np.arange(F.shape[0]) < n * n  # the triangle below the diagonal: u >= v
    wrong = np.where(lower, u[..., 1] - u[..., 0], u[..., 0] - u[..., 1])
    # A clipped point on the far side of the diagonal is nearest to the diagonal's projection.
    t = np.clip(((q - lo) / (hi - lo)).sum(-1) / 2, 0, 1)
    near = np.where((wrong > 0)[..., None], lo + t[..., None] * (hi - lo), c)
    d = (((q - near) ** 2).sum(-1) + height**2).astype(np.float32)
    order = bvh.ordering[::-1]
    for k in range(Q.shape[0]):
        ties = order[d[k, order] == d[k].min()][:8]
        assert nn[k] == ties[-1], (k, Q[k], ties, nn[k])


@pytest.mark.parametrize("itype", [np.int64, np.int32, np.uint16])
@pytest.mark.parametrize("n", [1, 255, 1000])
def test_arrays_by_rows_equal_arrays_by_columns(n, itype):
    """Row-major 3 x n arrays go to the device as they lie, others are transposed on the host: the same
    boxes, hierarchy and nearest triangles either way, and the same refusal of a bad index."""
    rng = np.random.default_rng(n)
    P = rng.uniform(-1, 1, (3, n + 2)).astype(np.float32)
    F = np.stack([np.arange(n), np.arange(n) + 1, np.arange(n) + 2]).astype(itype)
    Q = rng.uniform(-1, 1, (3, 77)).astype(np.float32)
    out = []
    for order in "CF":
        p, f, q = (np.array(a, order=order) for a in (P, F, Q))
        boxes = pbat.gpu.geometry.Aabb()
        boxes.construct(p, f)
        bvh = pbat.gpu.geometry.Bvh(n)
        bvh.build(np.array(boxes.min, order=order), np.array(boxes.max, order=order), [-1, -1, -1], [1, 1, 1])
        nn = bvh.point_triangle_nearest_neighbours(boxes, q, p, f)
        out.append((boxes.min, boxes.max, bvh.ordering, bvh.parent, nn))
        bad = np.array(F, order=order)
        bad[2, n - 1] = n + 2
        for call in (lambda: boxes.construct(p, bad), lambda: bvh.point_triangle_nearest_neighbours(boxes, q, p, bad)):
            with pytest.raises(_capi.PbgbError) as err:
                call()
            assert err.value.code == 1 and "out of range" in str(err.value)
        # The refusal leaves the hierarchy usable.
        np.testing.assert_array_equal(bvh.point_triangle_nearest_neighbours(boxes, q, p, f), nn)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def scan_without_bound(bvh, lo, hi, x, distance):
    """The nearest simplex as the query's depth-first scan leaves it: right child first, nodes passed over by
    their box alone, ties of the smallest distance kept in a list of 8 whose last entry stays."""
    t = bvh._topology()
    n = lo.shape[0]
    x = np.asarray(x, np.float32)

    def box(k):
        l, h = (t["ilo"][k], t["ihi"][k]) if k < n - 1 else (lo[t["inds"][k - n + 1]], hi[t["inds"][k - n + 1]])
        d = np.maximum(np.maximum(l - x, x - h), 0).astype(np.float64)
        return (d * d).sum()

    stack, ties, best = [0], [], np.inf
    while stack:
        k = stack.pop()
        if box(k) > best:
            continue
        if k < n - 1:
            stack += [t["child"][k][0], t["child"][k][1]]
            continue
        i = int(t["inds"][k - n + 1])
        d = distance(x, i)
        if d < best:
            best, ties = d, [i]
        elif d <= best and len(ties) < 8:
            ties.append(i)
    return ties[-1] if ties else -1


def boxes_and_tree(P, S):
    boxes = pbat.gpu.geometry.Aabb()
    boxes.construct(P.T, S.T)
    bvh = pbat.gpu.geometry.Bvh(S.shape[0])
    bvh.build(boxes, P.min(0) - 1, P.max(0) + 1)
    return boxes, bvh


def test_a_tetrahedron_on_a_line_is_its_own_nearest():
    """No volume: every point of the space is at distance zero by the face tests, also far from the box."""
    P = np.array([[0, 0, 0], [1, 0, 0], [2, 0, 0], [3, 0, 0]], np.float32)
    T = np.array([[0, 1, 2, 3]])
    boxes, bvh = boxes_and_tree(P, T)
    Q = np.array([[0.5, 0, 0], [-4, 0, 0], [1, 7, 0], [90, -3, 2]], np.float32)
    np.testing.assert_array_equal(bvh.point_tetrahedron_nearest_neighbours(boxes, Q.T, P.T, T.T), np.zeros(4, np.int32))


@pytest.mark.parametrize("n", [1, 3, 40])
def test_nearest_of_flat_tetrahedra_in_their_plane(n):
    """Coplanar corners: a query of the plane is inside every tetrahedron by the face tests, so the scan takes the
    first leaf it meets and the ties whose box holds the query."""
    rng = np.random.default_rng(n)
    P = np.concatenate([rng.integers(-64, 64, (4 * n, 2)), np.zeros((4 * n, 1))], 1).astype(np.float32)
    T = np.arange(4 * n).reshape(n, 4)
    boxes, bvh = boxes_and_tree(P, T)
    Q = np.concatenate([rng.integers(-256, 256, (200, 2)), np.zeros((200, 1))], 1).astype(np.float32)
    nn = bvh.point_tetrahedron_nearest_neighbours(boxes, Q.T, P.T, T.T)
    lo, hi = boxes.min.T, boxes.max.T
    expected = [scan_without_bound(bvh, lo, hi, q, lambda x, i: 0.0) for q in Q]
    np.testing.assert_array_equal(nn, expected)


@pytest.mark.parametrize("shift", [3.0, 64.0, -500.0])
def test_nearest_triangles_with_boxes_of_an_earlier_pose(shift):
    """The hierarchy was built before the triangles moved: what the scan returns depends on the boxes it passes
    over, and is never nothing."""
    n = 9
    i, j = (a.ravel() for a in np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij"))
    P = np.stack([i, j, 0.0 * i], 1).astype(np.float32)
    a, b = (c.ravel() for c in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    v = a * (n + 1) + b
    F = np.stack([v, v + n + 1, v + n + 2], 1)  # the half of each cell with u >= v
    boxes, bvh = boxes_and_tree(P, F)
    moved = P + np.array([shift, 0, 0], np.float32)
    Q = np.concatenate([moved[:40] + [0.5, 0.25, 0], P[:40] + [0.5, 0.25, 2.0]]).astype(np.float32)

    def distance(x, t):
        # Dyadic coordinates: exact.
        o = moved[F[t][0]].astype(np.float64)
        u, w = x[0] - o[0], x[1] - o[1]
        cu, cw = min(max(u, 0.0), 1.0), min(max(w, 0.0), 1.0)
        if cw > cu:
            cu = cw = min(max((u + w) / 2, 0.0), 1.0)
        return (u - cu) ** 2 + (w - cw) ** 2 + float(x[2]) ** 2

    nn = bvh.point_triangle_nearest_neighbours(boxes, Q.T, moved.T, F.T)
    lo, hi = boxes.min.T, boxes.max.T
    np.testing.assert_array_equal(nn, [scan_without_bound(bvh, lo, hi, q, distance) for q in Q])


@pytest.mark.parametrize("k", [3, 4])
@pytest.mark.parametrize("scale,offset,flat", [(1.0, 0.0, 1.0), (0.01, 30.0, 1.0), (1.0, 0.0, 1e-3), (100.0, -3e3, 1e-5)])
def test_the_bound_changes_no_pick(k, scale, offset, flat):
    """Random simplices, round and flat, queries near and far: the same picks as when the bound is off.  One
    simplex lies far from every query; with a corner moved out of its box no bound is trusted."""
    rng = np.random.default_rng(int(100 * scale) + k)
    n = 700
    c = rng.uniform(-1, 1, (n, 1, 3)) * scale
    d = rng.uniform(-1, 1, (n, k, 3)) * scale * 0.05 * np.array([1, flat, flat**0.5])
    P = (c + d).reshape(-1, 3) + offset
    P[-k:] = offset + scale * 1e3 + d[0]
    P = P.astype(np.float32)
    S = np.arange(n * k).reshape(n, k)
    boxes, bvh = boxes_and_tree(P, S)
    Q = offset + scale * rng.uniform(-1, 1, (3000, 3)) * 10.0 ** rng.uniform(-2, 1, (3000, 1))
    Q = np.concatenate([Q, P[rng.integers(0, (n - 1) * k, 500)]]).astype(np.float32)
    query = bvh.point_triangle_nearest_neighbours if k == 3 else bvh.point_tetrahedron_nearest_neighbours
    out = P.copy()
    out[-1] += scale
    np.testing.assert_array_equal(query(boxes, Q.T, P.T, S.T), query(boxes, Q.T, out.T, S.T))


@pytest.mark.parametrize("order", "CF")
@pytest.mark.parametrize("itype,bad", [(t, b) for t in (np.int64, np.uint64, np.uint32) for b in (2**32 + 2, 2**63 + 1, 2**32 - 1, -1)
                                       if np.iinfo(t).min <= b <= np.iinfo(t).max])
def test_wide_indices_are_checked_before_they_are_narrowed(itype, order, bad):
    """An index that is out of range is refused, whatever its low 32 bits are."""
    rng = np.random.default_rng(0)
    P = np.array(rng.uniform(-1, 1, (3, 9)).astype(np.float32), order=order)
    F = np.array(np.stack([np.arange(7), np.arange(7) + 1, np.arange(7) + 2]).astype(itype), order=order)
    boxes = pbat.gpu.geometry.Aabb()
    boxes.construct(P, F)
    bvh = pbat.gpu.geometry.Bvh(7)
    bvh.build(boxes, [-1, -1, -1], [1, 1, 1])
    nn = bvh.point_triangle_nearest_neighbours(boxes, P, P, F)
    wrong = F.copy(order="K")
    wrong[1, 3] = bad
    for call in (lambda: boxes.construct(P, wrong), lambda: bvh.point_triangle_nearest_neighbours(boxes, P, P, wrong)):
        with pytest.raises(_capi.PbgbError) as err:
            call()
        assert err.value.code == 1 and "out of range" in str(err.value)
    np.testing.assert_array_equal(bvh.point_triangle_nearest_neighbours(boxes, P, P, F), nn)


def test_threads_query_one_hierarchy():
    """Queries of different sizes from several threads at once, each against its own points: every thread gets
    what it gets alone."""
    rng = np.random.default_rng(5)
    n = 2000
    P = (rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    F = np.arange(3 * n).reshape(n, 3)
    boxes, bvh = boxes_and_tree(P, F)
    V, S = np.ascontiguousarray(P.T), np.ascontiguousarray(F.T)
    queries = [rng.uniform(-1, 1, (3, m)).astype(np.float32) for m in (1, 700, 5000, 60, 20000, 333, 9000, 2500)]
    # A hierarchy each for the answers; the one that is shared has no workspace yet and grows it while others query.
    expected = []
    for q in queries:
        _, own = boxes_and_tree(P, F)
        expected.append(own.point_triangle_nearest_neighbours(boxes, q, V, S))

    def work(k):
        return [bvh.point_triangle_nearest_neighbours(boxes, queries[k], V, S) for _ in range(20)]

    with ThreadPoolExecutor(len(queries)) as pool:
        for k, out in enumerate(pool.map(work, range(len(queries)))):
            for nn in out:
                np.testing.assert_array_equal(nn, expected[k])
