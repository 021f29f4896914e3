"""The bounds the locality sort keeps with an uploaded field are those its
positions reduce to."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["octree", "hash", "nearest"])
def test_sort_grid_is_that_of_the_positions(kind):
    P, T = W.kuhn_mesh(3, 0.2, 2)
    P = (P * np.array([2.0, 0.5, 1e-3], np.float32) - np.float32(0.3)).astype(np.float32)
    D = np.zeros((2, len(P), 3), np.float32)
    t = np.array([0.0, 1.0], np.float32)
    f = {"octree": lambda: jt.OctreeFEMTimeSeriesFieldOptimized(D, t, P, T),
         "hash": lambda: jt.FEMTimeSeriesField(D, t, P, T), "nearest": lambda: jt.TimeSeriesField(D, t, P)}[kind]()
    before = f.sort_grid(5)
    f.jt_field()
    after = f.sort_grid(5)
    assert list(before.origin) == list(after.origin) and list(before.inv_cell) == list(after.inv_cell)
