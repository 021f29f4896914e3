"""The filter records and pruned lists do something: on a conforming mesh almost
every tetrahedron is marked alone and has gradients, and pruning shortens the
lists; where tetrahedra overlap, those that an earlier one covers are not."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32 = np.float32
ALONE = 2


def _mesh(overlap):
    P, T = W.kuhn_mesh(8, 0.2, 3)
    if overlap:                            # every tetrahedron again, moved by a little, behind the first ones
        P = np.concatenate([P, P + np.random.default_rng(2).normal(0, 0.01, P.shape).astype(F32)])
        T = np.concatenate([T, T + len(P) // 2]).astype(np.int32)
    return P, T


def _words(buffer, at, n):
    raw = buffer.contiguous().view(-1).cpu().numpy().view(np.uint8)
    return raw[at:at + 32 * n].view(np.uint32).reshape(n, 8)


def _gradients(w):
    h = w[:, 3:8].copy().view(np.float16).reshape(len(w), 10)
    return np.any(h[:, :9] != 0, axis=1)


@pytest.mark.parametrize("overlap", [False, True])
def test_hash_grid(overlap):
    P, T = _mesh(overlap)
    f = jt.FEMTimeSeriesField(np.zeros((2, len(P), 3), F32), np.array([0, 1], F32), P, T, fem_grid_resolution=6)
    f.jt_field()
    w = _words(f._dev["filters"], 64 * len(T), len(T))
    alone = (w[:, 7] >> 16 & ALONE) != 0
    assert _gradients(w).mean() > 0.99
    half = len(T) // 2
    if overlap:
        assert alone[:half].mean() > 0.9 and alone[half:].mean() < 0.05
    else:
        assert alone.mean() > 0.9
    start = f._dev["pruned_start"].cpu().numpy()
    assert f._cfem.sub_elems == f._dev["pruned_elems"].data_ptr()
    assert 0 < start[-1] < 0.6 * f.fem_mesh._n_sub_entries


@pytest.mark.parametrize("overlap", [False, True])
def test_octree(overlap):
    P, T = _mesh(overlap)
    f = jt.OctreeFEMTimeSeriesFieldOptimized(np.zeros((2, len(P), 3), F32), np.array([0, 1], F32), P, T)
    f.jt_field()
    depth = f._cmesh.locator & 0xFF
    assert depth > 0
    up = lambda b: (b + 63) // 64 * 64  # noqa: E731
    faces = up(8 * f._cmesh.n_nodes) + 64
    slots = up(up(faces + (3 << depth) * 8) + (8 << 3 * depth))
    w = _words(f._dev["locator"], slots + 64 * len(T), len(T))
    alone = (w[:, 7] >> 16 & ALONE) != 0
    assert _gradients(w).mean() > 0.99
    if overlap:
        second = f.octree_mesh.elems[:len(T)] >= len(T) // 2
        assert alone[~second].mean() > alone[second].mean() and alone.mean() < 0.9
    else:
        assert alone.mean() > 0.9
