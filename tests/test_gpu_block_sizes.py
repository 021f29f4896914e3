"""The block size a tracking launch picks by itself changes no bit, at the sizes
where it changes and with blocks that end anywhere."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("n", [1, 63, 65, 9_728, 9_729, 38_913, 77_825, 116_735, 116_737, 150_001, 200_003, 311_297])
def test_default_blocks_give_the_bits_of_256(n):
    import torch
    g = [np.linspace(0, 1, k).astype(F32) for k in (9, 8, 7)]
    t = np.linspace(0, 0.2, 4).astype(F32)
    f = jt.StructuredTimeSeriesField(W.abc_snapshots(W.grid_nodes(*g), t), t, *g)
    x = torch.from_numpy(np.random.default_rng(1).random((n, 3)).astype(F32)).cuda()
    ends = [jt.create_tracker("rk4", f, jt.reflective_boundary(W.UNIT), record_final_only=True, block_size=b,
                              stage_fields=False).track_particles(x, (0.0, 0.08), 9, dt=0.01, return_device=True)
            for b in (0, 256)]
    assert torch.equal(*ends)
