"""Which blended fields the adjoint's backward gathers: the rule, and that node
records, quads and snapshot pairs give the same gradients (to the rounding
of their blends: a few 2^-24 a stage, over 11 steps far below 1e-4 of the
largest entry) on odd node counts and segments with a remainder."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import adjoint as A
from jaxtrace_gb300 import tracker as T
from jaxtrace_gb300 import workloads as W

F32 = np.float32


@pytest.mark.parametrize("n,steps,nodes,quads", [(100_000, 20, 96 ** 3, False), (300_000, 20, 96 ** 3, False),
                                                 (10_000, 60, 64 ** 3, False), (100_000, 20, 64 ** 3, False),
                                                 (300_000, 20, 64 ** 3, True), (1_048_576, 50, 64 ** 3, True),
                                                 (20_000, 20, 17 ** 3, False), (1_000_000, 20, 96 ** 3, True)])
def test_rule(n, steps, nodes, quads):
    assert A._quads_pay(n, steps, nodes) == quads


def test_small_forward_passes_are_turned_away_before_any_work(monkeypatch):
    g = np.linspace(0, 1, 33).astype(F32)
    s = A.AdjointRK4(np.linspace(0, 1, 4).astype(F32), g, g, g, "clamp")

    def looked(*a):
        raise AssertionError("the entries were looked at")
    monkeypatch.setattr(T, "_stage_entries", looked)
    assert s._blend_ahead(None, 20, np.zeros((20_000, 3), F32)) is None
    assert s._blend_ahead(None, 0, np.zeros((20_000, 3), F32)) is None
    with pytest.raises(AssertionError):
        monkeypatch.setattr(A, "_torch", lambda: None)
        s._blend_ahead(None, 50, np.zeros((1_000_000, 3), F32))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["periodic", "clamp"])
@pytest.mark.parametrize("dims,k", [((5, 7, 9), 4), ((5, 7, 9), 50), ((8, 4, 6), 3), ((3, 3, 3), 11)])
def test_every_layout_gives_the_gradients(monkeypatch, mode, dims, k):
    import torch
    g = [(np.arange(n) / n).astype(F32) if mode == "periodic" else np.linspace(0, 1, n).astype(F32) for n in dims]
    t = np.linspace(0, 0.2, 4).astype(F32)
    data = W.abc_snapshots(W.grid_nodes(*g), t)
    x = np.random.default_rng(1).random((500, 3)).astype(F32)
    cot = torch.from_numpy(np.random.default_rng(2).normal(size=x.shape).astype(F32)).cuda()
    bc = jt.periodic_boundary(W.UNIT) if mode == "periodic" else jt.reflective_boundary(W.UNIT)
    out = []
    for stage, quads in ((False, False), (True, False), (True, True)):
        monkeypatch.setattr(A, "_quads_pay", lambda *a, quads=quads: quads)
        s = A.AdjointRK4(t, *g, mode, bc, checkpoint_every=k, stage_fields=stage, sort_min_particles=100)
        x0 = torch.from_numpy(x).cuda().requires_grad_(True)
        U = torch.from_numpy(data.reshape(4, *dims, 3)).cuda().requires_grad_(True)
        xT = s(x0, U, (0.0, 0.22), 12, dt=0.02)
        out.append((xT.detach(), *torch.autograd.grad(xT, (x0, U), cot)))
    for o in out[1:]:
        assert torch.equal(o[0], out[0][0])
        for a, b in zip(o[1:], out[0][1:]):
            assert float((a - b).abs().max()) <= 1e-4 * float(b.abs().max())
