"""Optional device buffers are sized against the memory that can be had."""
import pytest
import torch

from jaxtrace_gb300.fields import room_for


@pytest.mark.parametrize("free,cached,size,fits", [(400, 0, 100, True), (400, 0, 101, False), (0, 400, 100, True),
                                                   (200, 200, 100, True), (200, 196, 100, False), (0, 0, 1, False)])
def test_free_and_cached_memory_count(monkeypatch, free, cached, size, fits):
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (free, 1000))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda device=None: 600)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda device=None: 600 - cached)
    assert room_for(size) == fits


@pytest.mark.gpu
def test_a_repeated_gradient_takes_the_same_buffer(monkeypatch):
    """The blocks a first gradient leaves with the allocator do not push the second
    one to another layout and another block."""
    import numpy as np

    import jaxtrace_gb300 as jt
    from jaxtrace_gb300 import adjoint as A
    monkeypatch.setattr(A, "_quads_pay", lambda *a: True)
    torch.cuda.empty_cache()
    g = (np.arange(32) / 32).astype(np.float32)
    s = A.AdjointRK4(np.linspace(0, 1, 3).astype(np.float32), g, g, g, "periodic", checkpoint_every=20)
    x = torch.rand(100, 3, device="cuda", requires_grad=True)
    U = torch.rand(3, 32, 32, 32, 3, device="cuda", requires_grad=True)
    stage = 3 * 20 * 32 ** 3 * 48
    total = 5 * stage
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d=None: (total - torch.cuda.memory_reserved(), total))
    layouts = []
    lib = A.L.load()
    monkeypatch.setattr(A.L, "load", lambda: Spy(lib, layouts))
    for _ in range(3):
        xT = s(x, U, (0.0, 0.2), 21, dt=0.01)
        torch.autograd.grad(xT.sum(), (x, U))
    assert set(layouts) == {A.L.JT_STORE_STAGE_F32Q}


class Spy:
    """The library, with the layout of every jt_stage_fields call written down."""

    def __init__(self, lib, layouts):
        self.lib, self.layouts = lib, layouts

    def __getattr__(self, name):
        f = getattr(self.lib, name)
        if name != "jt_stage_fields":
            return f

        def call(field, src, scales, n, storage, *rest):
            self.layouts.append(storage)
            return f(field, src, scales, n, storage, *rest)
        return call
