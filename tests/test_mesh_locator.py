"""The octree locator (jt_mesh_locator_build): its cells take the descent's
own moves, and the fields that use it return the bits of those that descend
node by node and gather the candidates through the element list."""
import ctypes as C

import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import _lib as L
from jaxtrace_gb300 import fields as F
from jaxtrace_gb300 import workloads as W
from test_octree_bfs import _bfs

F32 = np.float32


def _mesh(name):
    """(points, tets, max_elements_per_leaf, max_depth)"""
    P, T = W.kuhn_mesh({"pow2": 8, "odd": 5, "deep": 4, "cut": 6, "one": 1, "flat": 3, "sliver": 4, "offset": 4}[name],
                       0.2, 3)
    if name == "flat":        # a layer 1e-3 thick
        P = P * np.array([1, 1, 1e-3], F32)
    if name == "sliver":      # a few tetrahedra flattened onto their first face
        P = P.copy()
        P[T[::17, 3]] = (P[T[::17, 0]] + P[T[::17, 1]] + P[T[::17, 2]]) / 3 + F32(1e-6)
    if name == "offset":      # far from the origin: coarse float32 coordinates
        P = (P + F32(1000.25)).astype(F32)
    leaf, depth = {"deep": (1, 12), "cut": (1, 2), "pow2": (32, 12)}.get(name, (8, 12))
    return P.astype(F32), T, leaf, depth


def _queries(P, S, rng, n=3000):
    lo, hi = P.min(axis=0), P.max(axis=0)
    q = (lo + (hi - lo) * rng.uniform(-0.2, 1.2, (n, 3))).astype(F32)
    face = np.stack([rng.choice(S[a], n) for a in range(3)], axis=1)          # on faces and one float beside
    side = rng.integers(-1, 2, (n, 3))
    face = np.where(side < 0, np.nextafter(face, F32(-np.inf)), np.where(side > 0, np.nextafter(face, F32(np.inf)), face))
    pick = rng.integers(0, 2, (n, 3)).astype(bool)
    special = np.array([[np.nan, 0.1, 0.2], [np.inf, -np.inf, 0.3], [0.1, np.nan, np.nan], [-0.0, 0.0, -0.0]], F32)
    return np.concatenate([q, np.where(pick, face, q), P, special]).astype(F32)


@pytest.mark.parametrize("name", ["pow2", "odd", "deep", "cut", "one", "flat", "offset"])
def test_cells_take_the_descent_moves(name):
    P, T, leaf, depth = _mesh(name)
    m = jt.OctreeMesh(P, T, leaf, depth, build="host")
    desc, dtab = F.breadth_first_descent(m.nodes)
    D = min(int(m.info.max_tree_depth), m.max_depth, L.JT_MESH_LOCATOR_MAX_DEPTH)
    if D == 0:
        pytest.skip("a single leaf has no locator")
    S = F.locator_splits(m.nodes_min[0], m.nodes_max[0], D)
    for p in _queries(P, S, np.random.default_rng(5), 400):
        cell = [int(np.sum(S[a, 1:-1] <= p[a])) for a in range(3)]
        node = 0
        for d in range(D):                       # the moves of the cell's own path
            w = int(desc[node, 3].view(np.uint32))
            o = sum(((cell[a] >> (D - 1 - d)) & 1) << a for a in range(3))
            if not (w & 0xFF) >> o & 1:
                break
            node = (w >> 8) + bin(w & 0xFF & ((1 << o) - 1)).count("1")
        assert tuple(dtab[node]) == _bfs(desc, dtab, p, D)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["pow2", "odd", "deep", "cut", "one", "flat", "sliver", "offset"])
@pytest.mark.parametrize("storage,arith", [("f32", L.JT_ARITH_EXACT), ("f32", L.JT_ARITH_COMPENSATED),
                                           ("bf16", L.JT_ARITH_COMPENSATED)])
def test_field_values_are_the_descents(name, storage, arith):
    P, T, leaf, depth = _mesh(name)
    rng = np.random.default_rng(7)
    D = rng.normal(size=(3, len(P), 3)).astype(F32)
    f = jt.OctreeFEMTimeSeriesFieldOptimized(D, np.array([0, 0.5, 1], F32), P, T, max_elements_per_leaf=leaf,
                                             max_depth=depth, storage=storage)
    f.jt_field()
    depth_used = min(int(f.octree_mesh.info.max_tree_depth), depth, L.JT_MESH_LOCATOR_MAX_DEPTH)
    assert (f._cmesh.locator & 0xFF) == depth_used
    S = F.locator_splits(f.octree_mesh.nodes_min[0], f.octree_mesh.nodes_max[0], max(depth_used, 1))
    q = _queries(P, S, rng)
    # barycentrics near the tolerances: points of faces and edges, and vertices
    b = rng.dirichlet(np.ones(4), 3000)
    b[::3, 0] = 0.0
    b[1::3, 2] = 0.999999 * b[1::3, 2] + 1e-6
    b /= b.sum(axis=1, keepdims=True)
    q = np.concatenate([q, np.einsum("nk,nkc->nc", b, P[T[rng.integers(0, len(T), 3000)]].astype(np.float64))]).astype(F32)
    got = f.sample_at_positions(q, 0.3, arith=arith)
    loc, f._cmesh.locator = f._cmesh.locator, 0
    assert loc == 0 or depth_used > 0
    ref = f.sample_at_positions(q, 0.3, arith=arith)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


def test_locator_refusals():
    lib = L.load()
    assert lib.jt_mesh_locator_bytes(0, 1, 1) == lib.jt_mesh_locator_bytes(1, 1, 8) == 0
    with pytest.raises(ValueError, match="required"):
        L.check(lib.jt_mesh_locator_build(None, 1, None, None, None))


@pytest.mark.gpu
@pytest.mark.parametrize("name,integrator", [("pow2", "rk4"), ("odd", "rk4"), ("cut", "rk2"), ("sliver", "rk4"),
                                             ("offset", "euler"), ("overlap", "rk4")])
def test_tracks_are_the_descents(name, integrator):
    """A tracking run, whose evaluations start from the thread's last hit, on
    conforming meshes and on one whose tetrahedra overlap (each listed twice,
    the copy moved by a little, so that the first hit is not the only one)."""
    P, T, leaf, depth = _mesh("pow2" if name == "overlap" else name)
    if name == "overlap":
        rng = np.random.default_rng(2)
        P = np.concatenate([P, P + rng.normal(0, 0.01, P.shape).astype(F32)])
        T = np.concatenate([T, T + len(P) // 2]).astype(np.int32)[rng.permutation(2 * len(T))]
    rng = np.random.default_rng(11)
    lo, hi = P.min(axis=0), P.max(axis=0)
    D = (rng.normal(size=(3, len(P), 3)) * (hi - lo)).astype(F32)
    x0 = (lo + (hi - lo) * rng.uniform(size=(5000, 3))).astype(F32)
    ends = []
    for locator in (True, False):
        f = jt.OctreeFEMTimeSeriesFieldOptimized(D, np.array([0, 0.5, 1], F32), P, T, max_elements_per_leaf=leaf,
                                                 max_depth=depth)
        f.jt_field()
        if not locator:
            f._cmesh.locator = 0
        bc = jt.mixed_boundary((lo, hi), {"x": "periodic", "y": "reflective", "z": "periodic"})
        tr = jt.create_tracker(integrator, f, bc, record_final_only=True)
        ends.append(tr.track_particles(x0, (0.0, 0.6), 61, dt=0.01).positions[-1])
    assert np.array_equal(ends[0].view(np.uint32), ends[1].view(np.uint32))
