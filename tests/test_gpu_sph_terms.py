"""Single SPH terms, where no sum of many hides their rounding."""
import numpy as np
import pytest

from jaxtrace_gb300.density import SPHDensityEstimator

pytestmark = pytest.mark.gpu
F32 = np.float32


def _one_term(kind, lo, hi):
    """(q, term of one particle at q smoothing lengths as a share of the term at
    0) for queries that have that particle alone in their support, among many
    more in the same rows of cells."""
    import torch
    rng = np.random.default_rng(3)
    h = 0.02
    g = 0.5 + 0.143 * np.arange(-3, 4)
    q0 = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3).astype(F32)
    d = rng.normal(size=q0.shape)
    d *= (rng.uniform(lo, hi, len(q0)) * h / np.linalg.norm(d, axis=1))[:, None]
    near = (q0 + d).astype(F32)
    fill = rng.random((400_000, 3)).astype(F32)
    cell = 0.5 + 0.143 * np.rint((fill.astype(np.float64) - 0.5) / 0.143).clip(-3, 3)
    fill = fill[np.linalg.norm(fill - cell, axis=1) > (2.1 + hi) * h]     # outside the partner's support too
    P = np.concatenate([near, fill])
    s = SPHDensityEstimator(P, dimensions="3d", smoothing_length=h, kernel_type=kind, normalize=False)
    at = s._density_sum(torch.from_numpy(np.concatenate([q0, near])).cuda()).cpu().numpy()
    r = np.linalg.norm(near.astype(np.float64) - q0, axis=1) / np.float64(F32(h))
    return r, at[:len(q0)] / at[len(q0):]


@pytest.mark.parametrize("kind", ["cubic_spline", "wendland"])
def test_near_terms_round_once(kind):
    """Below q = 0.05 the kernel's float32 value is its last rounding, half a unit
    in the last place of [0.5, 1), and the rounding of q, which moves it by at
    most 10 q^2 (8 2^-24): 2^-25 and 1.2e-8.  Wendland's adds two products'
    and the slope's roundings of 1 - q: five more of 2^-24 and 20 q 2^-25."""
    r, got = _one_term(kind, 0.001, 0.05)
    if kind == "cubic_spline":
        want, tol = 1 - 1.5 * r ** 2 + 0.75 * r ** 3, 2.0 ** -25 + 1.2e-8
    else:
        want, tol = (1 - r) ** 4 * (1 + 4 * r), 6 * 2.0 ** -24
    assert np.abs(got - want).max() <= tol


def test_both_branches_of_the_spline():
    """Across q = 1: value 0.25 with slope -0.75; the rounding of q (8 2^-24) and
    four roundings of values up to 1 stay below 12 2^-24."""
    r, got = _one_term("cubic_spline", 0.9, 1.1)
    want = np.where(r <= 1, 1 - 1.5 * r ** 2 + 0.75 * r ** 3, 0.25 * (2 - r) ** 3)
    assert np.abs(got - want).max() <= 12 * 2.0 ** -24


@pytest.mark.parametrize("kind,reach", [("cubic_spline", 2.0), ("wendland", 1.0)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_masses_that_are_not_finite_in_pair_records(monkeypatch, kind, reach, bad):
    """Pair records take any mass, and a finite check costs no call a look at all
    masses: the sums that the particle reaches are not finite, the others are
    those without it, though their rows of cells hold it too (to 1e-5: the
    order of a cell's particles differs from run to run)."""
    import torch
    from jaxtrace_gb300 import density
    rng = np.random.default_rng(1)
    h = 0.05
    P = torch.from_numpy(rng.random((100_000, 3)).astype(F32)).cuda()
    q = P[:20_000].contiguous()
    m = rng.uniform(0.5, 2.0, len(P)).astype(F32)
    paired = []
    monkeypatch.setattr(density, "pair_records", lambda *a, f=density.pair_records: paired.append(1) or f(*a))
    sums = []
    for k in (None, 7, 8):                       # either half of a pair, by the cells' order
        if k is not None:
            m[k] = bad
        s = SPHDensityEstimator(P, dimensions="3d", smoothing_length=h, kernel_type=kind, masses=m, normalize=False)
        sums.append(s._density_sum(q).cpu().numpy())
    assert len(paired) == 3
    d = np.stack([np.linalg.norm((q - P[k]).double().cpu().numpy(), axis=1) for k in (7, 8)]) / np.float64(F32(h))
    for rho, near in zip(sums[1:], (d[0], d.min(axis=0))):
        inside, outside = near < reach - 1e-5, near > reach + 1e-5
        assert inside.any() and not np.isfinite(rho[inside]).any()
        assert np.allclose(rho[outside], sums[0][outside], rtol=1e-5)


@pytest.mark.parametrize("kind", ["cubic_spline", "wendland"])
@pytest.mark.parametrize("dims", [2, 3])
def test_rows_choose_the_loop(kind, dims):
    """Sparse rows keep the tested loop, whose sums are those of its terms in
    particle order, bit for bit; long ones take the other.  Cells are set
    here, so that one row holds them all or hardly any."""
    import ctypes as C

    import torch
    from jaxtrace_gb300 import _lib as L
    from jaxtrace_gb300 import density as D
    rng = np.random.default_rng(4)
    n, h = 6000, (0.05 if dims == 3 else 0.01)
    P = rng.random((n, 3)).astype(F32)
    if dims == 2:
        P[:, 2] = 0
    dev = torch.from_numpy(P).cuda()
    got = {}
    for cell in (1.0, 0.01):
        cl = D.CellList(dev, [0.0] * 3, [1.0, 1.0, 1.0 if dims == 3 else 0.0], cell, dims)
        out = {}
        for packed in (1, 2):
            m = torch.ones(n, device="cuda")
            rec = D.pair_records(cl.sorted, m) if packed == 2 else torch.cat([cl.sorted, m[:, None]], 1).contiguous()
            o = torch.empty(n, dtype=torch.float64, device="cuda")
            p = L.SphParams()
            p.dims, p.kernel = dims, D._SPH_KERNELS[kind]
            p.n_particles = p.n_queries = n
            p.radius, p.h_const, p.grid, p.packed = 3 * h, h, cl.grid, packed
            p.reach[:] = cl.reach(2 * h)
            p.particles, p.cell_end, p.queries, p.out = (t.data_ptr() for t in (rec, cl.cell_end, cl.sorted, o))
            L.check(L.load().jt_sph_density(C.byref(p), L.stream_ptr()))
            out[packed] = o.cpu().numpy()
        got[cell] = out
        assert np.allclose(out[1], out[2], rtol=1e-5)
    assert np.array_equal(got[0.01][1], got[0.01][2])          # one or two candidates a row: the same loop's terms
    assert not np.array_equal(got[1.0][1], got[1.0][2])        # thousands a row: the other


@pytest.mark.parametrize("lo,hi", [(0.05, 0.5), (0.5, 0.95), (1.05, 1.5), (1.5, 1.99)])
def test_terms_round_as_the_spline_of_the_tested_loop(lo, hi):
    """The rounding of q, at most 8 2^-24 of it, times the slope (at most 1 at
    q = 2/3), and four roundings of values up to 1."""
    r, got = _one_term("cubic_spline", lo, hi)
    want = np.where(r <= 1, 1 - 1.5 * r ** 2 + 0.75 * r ** 3, 0.25 * (2 - r) ** 3)
    assert np.abs(got - want).max() <= 12 * 2.0 ** -24
