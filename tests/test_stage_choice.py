"""When a float32 run blends its stage fields ahead: the rule, and that both
ways give the same bits for every integrator (RK2 and Euler leave schedule
entries unread, for which no field is blended)."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import _lib as L
from jaxtrace_gb300 import tracker as T
from jaxtrace_gb300 import workloads as W
from jaxtrace_gb300.schedule import build_schedule

F32 = np.float32


@pytest.mark.parametrize("code,read", [(L.JT_EULER, 1), (L.JT_RK2, 2), (L.JT_RK4, 3)])
def test_entries_that_are_not_read_get_no_field(code, read):
    steps = np.linspace(0, 0.11, 12).astype(F32)
    sched = build_schedule(steps, 0.01, code, np.linspace(0, 1, 5).astype(F32))
    host, uid = T._stage_entries(sched, 11, code)
    per = uid.reshape(11, 3)
    assert np.all(per[:, read - 1:] == per[:, read - 1:read])           # the unread ones repeat
    assert len(np.unique(per[:, :read], axis=0)) == 11
    a, b = host.reshape(11, 4), sched.reshape(11, 4)
    assert np.array_equal(a[:, :read], b[:, :read]) and np.array_equal(a[:, 3], b[:, 3])


@pytest.mark.parametrize("n,nodes,steps,ahead", [(10_000, 32 ** 3, 100, False), (300_000, 32 ** 3, 100, True),
                                                 (1_000_000, 128 ** 3, 100, False), (2_097_152, 128 ** 3, 100, True),
                                                 (16_777_216, 128 ** 3, 1000, True), (1000, 8, 10, False)])
def test_rule(n, nodes, steps, ahead):
    uid = np.arange(int(2.27 * steps))
    assert (T._stage_gain(n, steps, L.JT_RK4, uid, nodes) >= T.TrackerOptions().stage_min_gain) == ahead


@pytest.mark.gpu
@pytest.mark.parametrize("integrator", ["euler", "rk2", "rk4"])
@pytest.mark.parametrize("mode", ["periodic", "clamp", "nan"])
@pytest.mark.parametrize("n", [1, 77, 3000])
def test_both_ways_give_the_same_bits(integrator, mode, n):
    g = [(np.arange(k) / k).astype(F32) if mode == "periodic" else np.linspace(0, 1, k).astype(F32) for k in (9, 7, 4)]
    t = np.linspace(0, 0.2, 5).astype(F32)
    f = jt.StructuredTimeSeriesField(W.abc_snapshots(W.grid_nodes(*g), t), t, *g, mode)
    bc = jt.periodic_boundary(W.UNIT) if mode == "periodic" else jt.reflective_boundary(W.UNIT)
    x0 = np.random.default_rng(2).random((n, 3)).astype(F32)
    out = []
    for gain in (0.0, 1e30):
        tr = jt.create_tracker(integrator, f, bc, stage_min_gain=gain, stage_chunk=4, sort_every=5)
        out.append(tr.track_particles(x0, (0.0, 0.23), 24, dt=0.01).positions)
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
