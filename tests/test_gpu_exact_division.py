"""The exact arithmetic's division by the grid spacings: cell and weight of a
sampled point are those of the float32 quotient, for spacings of every kind of
significand and exponent, and points from far inside a cell to far outside."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import _lib as L

pytestmark = pytest.mark.gpu
F32 = np.float32


def _spacings():
    r = np.random.default_rng(0)
    some = [F32(1 / 127), F32(1 / 3), F32(0.1), F32(1.0), np.nextafter(F32(1), F32(2)), np.nextafter(F32(2), F32(0)),
            np.nextafter(F32(0.25), F32(1)), F32(3e-13), F32(2e12), F32(7e-12), F32(1e12), F32(1e-30), F32(1e30)]
    return some + [F32(v) for v in 2.0 ** r.uniform(-20, 20, 12) * r.uniform(1, 2, 12)]


@pytest.mark.parametrize("d", _spacings())
@pytest.mark.parametrize("origin", [0.0, 1.0])
def test_weights_are_those_of_the_quotient(d, origin):
    n = 33
    org = F32(origin) * d
    ax = (org + np.arange(n, dtype=F32) * d).astype(F32)
    step = F32(F32(ax[1]) - F32(ax[0]))                 # the field's own spacing
    if not (np.isfinite(ax).all() and step > 0):
        pytest.skip("no such grid in float32")
    v = (np.arange(n) % 2).astype(F32)
    data = np.zeros((1, n, 1, 1, 3), F32)
    data[0, :, 0, 0, 0] = v
    f = jt.StructuredTimeSeriesField(data, np.zeros(1, F32), ax, np.zeros(1, F32), np.zeros(1, F32), "clamp")
    r = np.random.default_rng(1)
    with np.errstate(over="ignore"):
        x = np.concatenate([org + step * F32(n) * r.random(400_000, dtype=F32),                       # inside
                            org + (step * 2.0 ** r.uniform(-100, 30, 50_000)).astype(F32),           # tiny and far
                            ax, np.nextafter(ax, F32(-np.inf)), np.nextafter(ax, F32(np.inf)),
                            np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-40, -1e-44], F32)]).astype(F32)
    p = np.zeros((len(x), 3), F32)
    p[:, 0] = x
    got = f.sample_at_positions(p, 0.0, arith=L.JT_ARITH_EXACT)[:, 0]
    with np.errstate(all="ignore"):
        q = np.clip((x - F32(ax[0])) / step, F32(0), F32(n - 1))
        fl = np.floor(q)
        w = q - fl
        i = np.nan_to_num(fl).astype(np.int64)
        ref = v[i] * (F32(1) - w) + v[np.minimum(i + 1, n - 1)] * w
    same = (got == ref) | (np.isnan(got) & np.isnan(ref))
    assert same.all(), (x[~same][:5], got[~same][:5], ref[~same][:5])
