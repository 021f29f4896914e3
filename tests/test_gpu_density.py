"""GPU density passes against the reference's golden vectors and the float64
oracle.  Tolerances: rtol 2e-5 (the reference computes in float32; the GPU
sums float32 cell/chunk partials in float64, uses the fast exponential and
skips KDE terms beyond 5 bandwidths along an axis, each below 4e-6)."""
import numpy as np
import pytest

import jaxtrace_gb300 as jt
from jaxtrace_gb300.density import KDEEstimator, SPHDensityEstimator
from oracle import density as OD

pytestmark = pytest.mark.gpu
F32 = np.float32


def test_kde_3d_grid(golden):
    g = golden("density")
    k = KDEEstimator(g["P"], bandwidth_rule="scott", resolution=12)
    assert abs(k.h - float(g["kde_h"])) < 1e-6 * k.h
    X, Y, Z, D = k.evaluate_3d()
    assert np.array_equal(X, g["kde3_X"]) and np.array_equal(Y, g["kde3_Y"]) and np.array_equal(Z, g["kde3_Z"])
    assert np.allclose(D, g["kde3_D"], rtol=2e-5, atol=1e-7)


def test_kde_2d_slab_grid(golden):
    g = golden("density")
    k = KDEEstimator(g["P"], bandwidth_rule="silverman", resolution=20, plane="xz", slab_position=0.5,
                     slab_thickness=0.3)
    X, Y, Z = k.evaluate_2d()
    assert np.array_equal(X, g["kde2_X"]) and np.array_equal(Y, g["kde2_Y"])
    assert np.allclose(Z, g["kde2_Z"], rtol=2e-5, atol=1e-7)


def test_kde_points(golden):
    g = golden("density")
    k = KDEEstimator(g["P"], bandwidth_rule="scott")
    assert np.allclose(k.evaluate(g["kde_q"]), g["kde_pts"], rtol=2e-5, atol=1e-9)


@pytest.mark.parametrize("kind", ["cubic_spline", "wendland", "gaussian"])
def test_sph_3d(golden, kind):
    g = golden("density")
    s = SPHDensityEstimator(g["P"], dimensions="3d", smoothing_length=0.08, kernel_type=kind)
    assert np.allclose(s.evaluate(g["P"]), g[f"sph3_{kind}"], rtol=2e-5, atol=1e-6)


def test_sph_2d_default_h(golden):
    g = golden("density")
    s = SPHDensityEstimator(g["P"], dimensions="2d", plane="xy", position=0.5, slab_thickness=0.4)
    assert abs(s._mean_h - float(g["sph2_default_h"])) < 1e-6
    assert np.allclose(s.evaluate(g["P"]), g["sph2_default"], rtol=2e-5, atol=1e-6)


def test_sph_adaptive(golden):
    g = golden("density")
    s = SPHDensityEstimator(g["P"][:400], dimensions="3d", adaptive=True, n_neighbors=16)
    assert np.allclose(s.smoothing_lengths.cpu().numpy(), g["sph3_adaptive_h"], rtol=1e-6)
    assert np.allclose(s.evaluate(g["P"][:400]), g["sph3_adaptive"], rtol=2e-5, atol=1e-6)


def test_sph_and_kde_at_scale_vs_oracle():
    """200k uniform particles: every 97th query against the float64 brute force."""
    rng = np.random.default_rng(5)
    P = rng.random((200_000, 3)).astype(F32)
    s = SPHDensityEstimator(P, dimensions="3d", smoothing_length=0.02, normalize=False)
    rho = s.evaluate(P)
    sub = np.arange(0, len(P), 97)
    ref = OD.sph_sum(P[sub], P, np.float32(0.02))
    assert np.allclose(rho[sub], ref, rtol=2e-5)
    k = KDEEstimator(P, bandwidth=0.03)
    q = rng.random((500, 3)).astype(F32)
    assert np.allclose(k.evaluate(q), OD.kde_mean(q, P, 0.03), rtol=2e-5)


@pytest.mark.parametrize("n,res,scale", [(2, (8, 8, 8), 1.0), (3, (1, 9, 17), 1.0), (255, (7, 8, 9), 0.1),
                                         (1025, (16, 15, 3), 0.3), (40_000, (20, 33, 12), 0.02), (9000, (24, 24, 24), 1.0)])
@pytest.mark.parametrize("cutoff", [5.0, 6.5])
def test_kde_3d_grid_tiles_and_row_lists(n, res, scale, cutoff):
    """Grids that end inside a tile, chunks and row lists that end anywhere (a
    small bandwidth cuts 2^7 cells per axis, thousands of rows a tile), clumped
    particles.  Terms dropped lie beyond 1.2 cutoffs: below n exp(-18) in all,
    which is far below the 2e-5 of the largest sum allowed."""
    rng = np.random.default_rng(n)
    P = (0.5 + 0.2 * rng.normal(size=(n, 3)) * np.array([1.0, 0.3, 1.0])).astype(F32)
    k = KDEEstimator(P, bandwidth=0.1 * scale + 0.01, resolution=res, cutoff_sigmas=cutoff, normalize=False,
                     bounds=((0.0, 1.0), (-0.2, 1.2), (0.1, 0.9)))
    X, Y, Z, D = k.evaluate_3d()
    q = np.stack([X, Y, Z], axis=-1).reshape(-1, 3)
    ref = OD.kde_mean(q, P, k.h).reshape(D.shape)
    assert np.allclose(D, ref, rtol=2e-5, atol=2e-5 * ref.max())


@pytest.mark.parametrize("kind", ["cubic_spline", "wendland"])
@pytest.mark.parametrize("dims", ["2d", "3d"])
@pytest.mark.parametrize("n,h", [(2, 0.5), (3, 0.02), (501, 0.15), (20_000, 0.03), (3000, 1e-3)])
def test_sph_sums_without_a_support_test(kind, dims, n, h):
    """Rows that start and end inside a pair of particles, twins (distance 0),
    few and many candidates, against the float64 sum.  A term is off by a few
    2^-24 of the kernel's height; 2e-5 of the sum covers one term alone."""
    rng = np.random.default_rng(n)
    P = rng.random((n, 3)).astype(F32)
    P[n // 2:n // 2 + n // 8] = P[:n // 8]
    m = rng.uniform(0.5, 2.0, n).astype(F32)
    s = SPHDensityEstimator(P, dimensions=dims, smoothing_length=h, kernel_type=kind, masses=m, normalize=False,
                            slab_thickness=4.0)
    q = np.concatenate([P[:300], rng.random((100, 3)).astype(F32)])
    rho = s.evaluate(q)
    a, b = (q, P) if dims == "3d" else (q[:, :2], P[:, :2])
    r = np.sqrt(((a[:, None].astype(np.float64) - b[None]) ** 2).sum(-1)) / np.float64(F32(h))
    hh = np.float64(F32(h))
    if kind == "cubic_spline":
        w = np.where(r <= 1, 1 - 1.5 * r ** 2 + 0.75 * r ** 3, 0.25 * np.clip(2 - r, 0, None) ** 3)
        w *= 10 / (7 * np.pi * hh ** 2) if dims == "2d" else 1 / (np.pi * hh ** 3)
    else:
        w = np.clip(1 - r, 0, None) ** 4 * (1 + 4 * r)
        w *= 7 / (np.pi * hh ** 2) if dims == "2d" else 21 / (2 * np.pi * hh ** 3)
    ref = (w * m[None]).sum(1)
    assert np.allclose(rho, ref, rtol=2e-5, atol=2e-5 * ref.max())


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_sph_particles_that_are_not_finite_stay_where_they_reach(bad):
    rng = np.random.default_rng(1)
    P = rng.random((2000, 3)).astype(F32)
    m = np.ones(2000, F32)
    q = rng.random((200, 3)).astype(F32)
    good = SPHDensityEstimator(P, dimensions="3d", smoothing_length=0.05, masses=m, normalize=False).evaluate(q)
    m[7] = bad
    rho = SPHDensityEstimator(P, dimensions="3d", smoothing_length=0.05, masses=m, normalize=False).evaluate(q)
    near = np.linalg.norm(q.astype(np.float64) - P[7], axis=1) < 0.1
    assert np.allclose(rho[~near], good[~near], rtol=2e-5) and not np.isfinite(rho[near]).any()
