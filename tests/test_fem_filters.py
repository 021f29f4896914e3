"""The hash-grid field with filter records and hints returns the bits of the
plain list scan, on conforming, odd, flattened, distant and overlapping meshes."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300 import _lib as L
from test_mesh_locator import _mesh

pytestmark = pytest.mark.gpu
F32 = np.float32
NAMES = ["pow2", "odd", "one", "flat", "sliver", "offset", "overlap", "planar"]


def _case(name):
    if name == "overlap":
        P, T, _, _ = _mesh("pow2")
        rng = np.random.default_rng(2)
        P = np.concatenate([P, P + rng.normal(0, 0.01, P.shape).astype(F32)])
        T = np.concatenate([T, T + len(P) // 2]).astype(np.int32)[rng.permutation(2 * len(T))]
        return P, T
    if name == "planar":      # no volume at all: one hash cell thick
        P, T, _, _ = _mesh("odd")
        P = P.copy()
        P[:, 2] = 0.5
        return P, T
    P, T, _, _ = _mesh(name)
    return P, T


def _plain(f):
    """The field without filters, on the mesh's own sub-cell lists."""
    f.jt_field()
    assert f._cfem.sub_div & L.JT_FEM_FILTERS
    f._cfem.sub_div &= ~L.JT_FEM_FILTERS
    h = f.fem_mesh
    if h.sub_div:
        f._cfem.sub_start, f._cfem.sub_elems = h.dev["sub_start"].data_ptr(), h.dev["sub_elems"].data_ptr()
    return f


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("storage,arith", [("f32", L.JT_ARITH_EXACT), ("f32", L.JT_ARITH_COMPENSATED),
                                           ("f16", L.JT_ARITH_COMPENSATED)])
def test_field_values_are_the_scans(name, storage, arith):
    P, T = _case(name)
    rng = np.random.default_rng(7)
    D = rng.normal(size=(3, len(P), 3)).astype(F32)
    t = np.array([0, 0.5, 1], F32)
    lo, hi = P.min(axis=0), P.max(axis=0)
    b = rng.dirichlet(np.ones(4), 4000)
    b[::3, 0] = 0.0
    b[1::3, 2] = 0.999999 * b[1::3, 2] + 1e-6
    b /= b.sum(axis=1, keepdims=True)
    q = np.concatenate([lo + (hi - lo) * rng.uniform(-0.1, 1.1, (4000, 3)), P,
                        np.einsum("nk,nkc->nc", b, P[T[rng.integers(0, len(T), 4000)]].astype(np.float64)),
                        [[np.nan, 0.1, 0.2], [np.inf, 0.0, 0.1], lo, hi]]).astype(F32)
    make = lambda: jt.FEMTimeSeriesField(D, t, P, T, fem_grid_resolution=6, storage=storage)  # noqa: E731
    got = make().sample_at_positions(q, 0.3, arith=arith)
    ref = _plain(make()).sample_at_positions(q, 0.3, arith=arith)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("sub_div", [0, 3, None])
def test_tracks_are_the_scans(name, sub_div):
    P, T = _case(name)
    rng = np.random.default_rng(11)
    lo, hi = P.min(axis=0), P.max(axis=0)
    ext = np.maximum(hi - lo, F32(1e-3))
    D = (rng.normal(size=(3, len(P), 3)) * ext).astype(F32)
    x0 = (lo + ext * rng.uniform(size=(4000, 3))).astype(F32)
    t = np.array([0, 0.5, 1], F32)
    bc = jt.mixed_boundary((lo, lo + ext), {"x": "periodic", "y": "reflective", "z": "periodic"})
    ends = []
    for plain in (False, True):
        f = jt.FEMTimeSeriesField(D, t, P, T, fem_grid_resolution=6, sub_div=sub_div)
        tr = jt.create_tracker("rk4", _plain(f) if plain else f, bc, record_final_only=True)
        ends.append(tr.track_particles(x0, (0.0, 0.6), 61, dt=0.01).positions[-1])
    assert np.array_equal(ends[0].view(np.uint32), ends[1].view(np.uint32))
