"""The optional lookup records of mesh and scattered-node fields are built once the
evaluations asked for would have paid for them, and change no bit."""
import numpy as np
import pytest
import torch

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import _lib as L
from jaxtrace_gb300 import fields as F
from jaxtrace_gb300 import workloads as W

F32 = np.float32


class _Fake(F._DeviceField):
    _records, _records_cost, _records_gain = False, 1000.0, (10.0, 0.5)
    _cfield, builds = None, 0

    def _device(self):
        pass

    def _build_records(self):
        self.builds += 1


def test_rule(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    f = _Fake()
    for k in range(9):                    # 10 chains of 10 us and 100 evaluations of 0.5 us: 110 us each
        f._field_for(2, 10)
        assert f.builds == 0
    f._field_for(2, 10)
    f._field_for(2, 10)
    f.jt_field()
    assert f.builds == 1
    f = _Fake()
    f._field_for(1000, 2)                 # one launch that pays
    assert f.builds == 1
    f = _Fake()
    f.jt_field()                          # asked for
    assert f.builds == 1


def test_nothing_is_built_into_a_graph(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    f = _Fake()
    f._field_for(10 ** 9, 100)
    assert f.builds == 0
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    f._field_for(1, 1)
    assert f.builds == 1


def _field(kind, storage="f32"):
    P, T = W.kuhn_mesh(9, 0.2, 3)
    rng = np.random.default_rng(1)
    D = rng.normal(size=(3, len(P), 3)).astype(F32)
    t = np.array([0, 0.5, 1], F32)
    if kind == "nearest":
        return jt.TimeSeriesField(D, t, P, storage=storage)
    return {"octree": jt.OctreeFEMTimeSeriesFieldOptimized, "hash": jt.FEMTimeSeriesField}[kind](D, t, P, T, storage=storage)


def _has(f, kind):
    return bool({"octree": lambda: f._cmesh.locator, "nearest": lambda: f._cnear.storage & L.JT_NEAREST_LISTS,
                 "hash": lambda: f._cfem.sub_div & L.JT_FEM_FILTERS}[kind]())


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["octree", "hash", "nearest"])
def test_probe_run_and_graph(kind):
    f = _field(kind)
    q = np.random.default_rng(2).uniform(-0.1, 1.1, (3000, 3)).astype(F32)
    plain = f.sample_at_positions(q, 0.3)
    held = f.memory_usage_mb()
    assert not _has(f, kind)              # a probe builds none
    tr = jt.create_tracker("rk4", f, jt.periodic_boundary(W.UNIT), record_final_only=True)
    batch = tr.ensemble_batch([q[:500], q[500:900]], [0.0, 0.2], 9, dt=0.01)
    batch.run()
    first = batch.pos.clone()
    assert not _has(f, kind)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):             # a pass captured on the plain field
        eng = batch._pass()
    f._saved = f._records_cost
    tr.track_particles(q, (0.0, 0.1), 11, dt=0.01)
    assert _has(f, kind) and f.memory_usage_mb() > held
    assert np.array_equal(f.sample_at_positions(q, 0.3).view(np.uint32), plain.view(np.uint32))
    junk = [torch.full((1 << 20,), -1, dtype=torch.int32, device="cuda") for _ in range(8)]   # over freed memory
    batch.pos.zero_()
    g.replay()                            # reads what it was captured on
    assert torch.equal(batch.pos, first) and len(junk) == 8 and eng is not None
    batch.run()
    assert torch.equal(batch.pos, first)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["octree", "hash", "nearest"])
def test_captured_batches_and_descriptors_have_them(kind):
    f = _field(kind, "bf16")
    tr = jt.create_tracker("rk4", f, jt.periodic_boundary(W.UNIT))
    q = np.random.default_rng(2).random((300, 3)).astype(F32)
    batch = tr.ensemble_batch([q], [0.0], 5, dt=0.01)
    assert not _has(f, kind)
    batch.capture().run()
    assert _has(f, kind)
    f = _field(kind)
    f.jt_field()
    assert _has(f, kind)
