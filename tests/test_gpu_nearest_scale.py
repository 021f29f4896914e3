"""The nearest node at any scale of the positions: candidate lists, and none where
squared distances leave float32's normal range."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("scale", [1e-22, 1e-21, 1e-20, 1e-18, 1e-15, 1e-12, 1e-6, 1e6, 1e15, 1e18, 1e19])
@pytest.mark.parametrize("flat", [False, True])
def test_search_is_the_argmin(scale, flat):
    rng = np.random.default_rng(3)
    ext = np.array([1.0, 1.0, 1e-9 if flat else 1.0]) * scale
    P = (rng.uniform(size=(3000, 3)) * ext).astype(F32)
    D = np.zeros((1, len(P), 3), F32)
    D[0, :, 0] = np.arange(len(P))
    q = (rng.uniform(-0.05, 1.05, (2000, 3)) * ext).astype(F32)
    with np.errstate(all="ignore"):
        d = q[:, None, :] - P[None]
        ref = np.argmin((d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2], axis=1)
    f = jt.TimeSeriesField(D, np.zeros(1, F32), P)
    for _ in range(2):                     # through the rings, then with every record
        assert np.array_equal(f.sample_at_positions(q, 0.0)[:, 0].astype(np.int64), ref)
        f.jt_field()
