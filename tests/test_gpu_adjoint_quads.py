"""The adjoint's blended fields: node counts that are odd, every bounds mode,
segments with a remainder; forward on quads or on pairs, backward on quads or
on pairs.  Positions are the same bits; gradients agree to float32 rounding
(the pair path blends the corners with another rounding: a few 2^-24 a stage,
over 11 steps far below 1e-4 of the largest entry)."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import tracker as T
from jaxtrace_gb300 import workloads as W
from jaxtrace_gb300.adjoint import AdjointRK4

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("mode", ["periodic", "clamp"])
@pytest.mark.parametrize("dims", [(5, 7, 9), (8, 4, 6), (3, 3, 2)])
@pytest.mark.parametrize("k", [4, 50])
def test_quads_give_the_pair_gradients(monkeypatch, mode, dims, k):
    import torch
    g = [(np.arange(n) / n).astype(F32) if mode == "periodic" else np.linspace(0, 1, n).astype(F32) for n in dims]
    t = np.linspace(0, 0.2, 4).astype(F32)
    data = W.abc_snapshots(W.grid_nodes(*g), t)
    x = np.random.default_rng(1).random((500, 3)).astype(F32)
    cot = torch.from_numpy(np.random.default_rng(2).normal(size=x.shape).astype(F32)).cuda()
    bc = jt.periodic_boundary(W.UNIT) if mode == "periodic" else jt.reflective_boundary(W.UNIT)
    out = []
    for stage, gain in ((False, 0.0), (True, 0.0), (True, 2.0)):
        monkeypatch.setattr(T, "_stage_gain", lambda *a, gain=gain: gain)
        s = AdjointRK4(t, *g, mode, bc, checkpoint_every=k, stage_fields=stage, sort_min_particles=100)
        x0 = torch.from_numpy(x).cuda().requires_grad_(True)
        U = torch.from_numpy(data.reshape(4, *dims, 3)).cuda().requires_grad_(True)
        xT = s(x0, U, (0.0, 0.22), 12, dt=0.02)
        out.append((xT.detach(), *torch.autograd.grad(xT, (x0, U), cot)))
    for o in out[1:]:
        assert torch.equal(o[0], out[0][0])
        for a, b in zip(o[1:], out[0][1:]):
            assert float((a - b).abs().max()) <= 1e-4 * float(b.abs().max())
