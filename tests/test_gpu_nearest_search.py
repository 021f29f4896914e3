"""The nearest-node search against the float32 argmin over all nodes: lattices
whose cell centres tie, twins, thin and distant node sets, queries far outside
and not finite; and tracks, whose evaluations start from the thread's last
node, against the oracle's brute force."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
import oracle

pytestmark = pytest.mark.gpu
F32 = np.float32


def _nodes(kind, rng):
    if kind == "lattice":
        g = np.arange(9, dtype=F32) / F32(8)
        return np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    if kind == "twins":       # every node three times
        return np.repeat(rng.uniform(size=(400, 3)).astype(F32), 3, axis=0)[rng.permutation(1200)]
    if kind == "clusters":    # empty cells around dense ones
        c = rng.uniform(size=(7, 3))
        return (c[rng.integers(0, 7, 2000)] + rng.normal(0, 1e-3, (2000, 3))).astype(F32)
    if kind == "plane":
        return np.concatenate([rng.uniform(size=(900, 2)), np.full((900, 1), 0.25)], axis=1).astype(F32)
    if kind == "line":
        return (np.linspace(0, 1, 257)[:, None] * np.array([[1.0, 0.0, 0.0]])).astype(F32)
    if kind == "offset":
        return (1000.0 + rng.uniform(size=(1500, 3)) * np.array([1, 1, 1e-2])).astype(F32)
    if kind == "one":
        return np.array([[0.3, 0.4, 0.5]], F32)
    return rng.uniform(size=(3000, 3)).astype(F32)


KINDS = ["random", "lattice", "twins", "clusters", "plane", "line", "offset", "one"]


@pytest.mark.parametrize("kind", KINDS)
def test_search_is_the_argmin(kind):
    rng = np.random.default_rng(3)
    P = _nodes(kind, rng)
    N = len(P)
    D = np.zeros((1, N, 3), F32)
    D[0, :, 0] = np.arange(N)               # the value is the node's number
    f = jt.TimeSeriesField(D, np.zeros(1, F32), P)
    lo, hi = P.min(axis=0), P.max(axis=0)
    ext = np.maximum(hi - lo, F32(1e-2))
    q = (lo + ext * rng.uniform(-0.3, 1.3, (1500, 3))).astype(F32)
    far = (lo + ext * rng.normal(0, 300.0, (60, 3))).astype(F32)
    mid = ((P[rng.integers(0, N, 500)] + P[rng.integers(0, N, 500)]) * F32(0.5)).astype(F32)
    odd = np.array([[1e25, 0, 0], [-1e30, 1e30, 0.1], [0.2, 3e38, 0.1], [np.inf, 0, 0]], F32)
    q = np.concatenate([q, far, mid, P[:500], odd])
    with np.errstate(over="ignore", invalid="ignore"):
        d = q[:, None, :] - P[None]
        ref = np.argmin((d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2], axis=1)
    got = f.sample_at_positions(q, 0.0)[:, 0]
    assert np.array_equal(got.astype(np.int64), ref)
    assert f.sample_at_positions(np.full((1, 3), np.nan, F32), 0.0)[0, 0] == 0.0


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("integrator", ["rk4", "euler"])
def test_tracks_are_the_oracles(kind, integrator):
    rng = np.random.default_rng(4)
    P = _nodes(kind, rng)
    lo, hi = P.min(axis=0), P.max(axis=0)
    ext = np.maximum(hi - lo, F32(1e-2))
    D = (rng.normal(size=(3, len(P), 3)) * ext).astype(F32)
    times = np.array([0, 0.5, 1], F32)
    x0 = (lo + ext * rng.uniform(size=(600, 3))).astype(F32)
    f = jt.TimeSeriesField(D, times, P)
    got = jt.create_tracker(integrator, f, jt.no_boundary(), record_final_only=True) \
        .track_particles(x0, (0.0, 0.4), 41, dt=0.01).positions[-1]
    code = {"rk4": "rk4", "euler": "euler"}[integrator]
    ref, _, _ = oracle.track(oracle.NearestSpec(D, times, P), oracle.BoundarySpec(kinds=("none",) * 3), x0,
                             np.linspace(0, 0.4, 41, dtype=F32), 0.01, integrator=code)
    assert np.array_equal(got.view(np.uint32), np.asarray(ref, F32).view(np.uint32))
