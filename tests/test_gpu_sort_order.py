"""The z-first Morton order of the locality sort: slots in the order of its
keys, positions, Kahan terms and ids moved together, and back."""
import ctypes as C

import numpy as np
import pytest

from jaxtrace_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 257, 100_003])
@pytest.mark.parametrize("bits", [1, 4, 7])
@pytest.mark.parametrize("again", [False, True])
def test_records_move_together_in_key_order(n, bits, again):
    import torch
    g = L.SortGrid()
    g.origin[:] = [0.1, 0.0, -0.2]
    g.inv_cell[:] = [float(1 << bits), float(1 << bits) * 0.8, float(1 << bits) * 0.7]
    g.bits, g.order = bits, L.JT_ORDER_MORTON_Z
    lib = L.load()
    x = torch.rand((n, 3), device="cuda")
    c = torch.rand((n, 3), device="cuda")
    ids_in = torch.randperm(n, device="cuda").to(torch.int32) if again else None
    ws = torch.empty(int(lib.jt_cell_sort_workspace_bytes(n, bits)), dtype=torch.uint8, device="cuda")
    out, cout = torch.empty_like(x), torch.empty_like(c)
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    L.check(lib.jt_cell_sort(C.byref(g), n, L.ptr(x), L.ptr(c), L.ptr(ids_in), L.ptr(out), L.ptr(cout), L.ptr(ids),
                             L.ptr(ws), ws.numel(), L.stream_ptr()))
    src = ids.long() if ids_in is None else torch.argsort(ids_in.long())[ids.long()]
    assert torch.equal(torch.sort(src).values, torch.arange(n, device="cuda"))
    assert torch.equal(out, x[src]) and torch.equal(cout, c[src])
    p = out.cpu().numpy()
    cell = np.clip(np.floor((p - np.array(g.origin[:], np.float32)) * np.array(g.inv_cell[:], np.float32)), 0,
                   (1 << bits) - 1).astype(np.int64)
    key = sum(((cell[:, a] >> b) & 1) << (3 * b + 2 - a) for a in range(3) for b in range(bits))
    assert np.all(np.diff(key) >= 0)
