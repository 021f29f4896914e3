"""Sides of the rule for blending ahead, next to where it changes (measured times
stand beside the rule)."""
import numpy as np
import pytest

from jaxtrace_gb300 import _lib as L
from jaxtrace_gb300 import tracker as T


@pytest.mark.parametrize("n,nodes,steps,ahead", [(30_000, 32 ** 3, 100, False), (100_000, 32 ** 3, 100, True),
                                                 (100_000, 32 ** 3, 20, False), (400_000, 17 ** 3, 20, False),
                                                 (1_000_000, 17 ** 3, 20, True), (1_000_000, 128 ** 3, 100, False),
                                                 (400_000, 64 ** 3, 100, True)])
def test_rule(n, nodes, steps, ahead):
    uid = np.arange(int(2.31 * steps))
    assert (T._stage_gain(n, steps, L.JT_RK4, uid, nodes) >= T.TrackerOptions().stage_min_gain) == ahead
