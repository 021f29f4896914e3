"""When a run sorts its particles by cell by default."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import workloads as W

F32 = np.float32


def _tracker(kind):
    t = np.array([0, 1], F32)
    if kind == "grid":
        g = np.linspace(0, 1, 4).astype(F32)
        f = jt.StructuredTimeSeriesField(np.zeros((2, 64, 3), F32), t, g, g, g)
    else:
        P, _ = W.kuhn_mesh(2, 0.2, 2)
        f = jt.TimeSeriesField(np.zeros((2, len(P), 3), F32), t, P)
    return jt.create_tracker("rk4", f, jt.no_boundary())


@pytest.mark.parametrize("kind,n,steps,every", [("grid", 1 << 17, 1000, 0), ("grid", 1 << 18, 4, 100),
                                                ("nodes", (1 << 17) - 1, 1000, 0), ("nodes", 132_000, 8, 0),
                                                ("nodes", 200_000, 8, 0), ("nodes", 200_000, 16, 32),
                                                ("nodes", 200_003, 50, 32), ("nodes", 1 << 18, 4, 32)])
def test_default(kind, n, steps, every):
    assert _tracker(kind)._sort_every(n, steps) == every
