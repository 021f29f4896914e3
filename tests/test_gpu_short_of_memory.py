"""Mesh and scattered-node fields without room for their optional records work
as before and give the same bits."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import _lib as L
from jaxtrace_gb300 import fields as F
from jaxtrace_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32 = np.float32


def _make(kind, P, T, D, t):
    if kind == "nearest":
        return jt.TimeSeriesField(D, t, P)
    return {"octree": jt.OctreeFEMTimeSeriesFieldOptimized, "hash": jt.FEMTimeSeriesField}[kind](D, t, P, T)


def _flags(f, kind):
    f.jt_field()
    return {"octree": lambda: f._cmesh.locator, "nearest": lambda: f._cnear.storage & L.JT_NEAREST_LISTS,
            "hash": lambda: f._cfem.sub_div & L.JT_FEM_FILTERS}[kind]()


@pytest.mark.parametrize("kind", ["octree", "hash", "nearest"])
def test_fields_without_room(monkeypatch, kind):
    import torch
    P, T = W.kuhn_mesh(9, 0.2, 3)
    rng = np.random.default_rng(1)
    D = rng.normal(size=(3, len(P), 3)).astype(F32)
    t = np.array([0, 0.5, 1], F32)
    q = rng.uniform(-0.1, 1.1, (5000, 3)).astype(F32)
    f = _make(kind, P, T, D, t)
    assert _flags(f, kind)
    want = f.sample_at_positions(q, 0.3)
    with monkeypatch.context() as m:
        m.setattr(torch.cuda, "mem_get_info", lambda device=None: (0, 1 << 30))
        m.setattr(torch.cuda, "memory_reserved", lambda device=None: 0)
        m.setattr(torch.cuda, "memory_allocated", lambda device=None: 0)
        f = _make(kind, P, T, D, t)
        assert not _flags(f, kind)
        got = f.sample_at_positions(q, 0.3)
        tr = jt.create_tracker("rk4", f, jt.periodic_boundary(W.UNIT), record_final_only=True)
        tr.track_particles(q[:100], (0.0, 0.1), 11, dt=0.01)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("room", [1, 2])
def test_hash_grid_with_room_for_some(monkeypatch, room):
    """Filters without pruned lists, where one or both of the lists' arrays do not fit."""
    P, T = W.kuhn_mesh(9, 0.2, 3)
    rng = np.random.default_rng(1)
    D = rng.normal(size=(3, len(P), 3)).astype(F32)
    t = np.array([0, 0.5, 1], F32)
    q = rng.uniform(-0.1, 1.1, (5000, 3)).astype(F32)
    f = _make("hash", P, T, D, t)
    f.jt_field()
    want = f.sample_at_positions(q, 0.3)
    pruned = f._cfem.sub_elems
    asked = []
    monkeypatch.setattr(F, "room_for", lambda n, device=None: asked.append(n) or len(asked) <= 1 + room)
    f = _make("hash", P, T, D, t)
    f.jt_field()
    assert len(asked) == 2 + room and f._cfem.sub_div & L.JT_FEM_FILTERS
    assert f._cfem.sub_elems == f.fem_mesh.dev["sub_elems"].data_ptr() != pruned
    got = f.sample_at_positions(q, 0.3)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
