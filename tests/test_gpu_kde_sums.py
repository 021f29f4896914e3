"""What the 3-D KDE grid kernel sums, and in how many bits."""
import numpy as np
import pytest

from jaxtrace_gb300.density import KDEEstimator

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("n", [1003, 2047, 5001, 40_009])
def test_float32_sums_cover_few_particles(n):
    """Terms of 16 significant bits: float32 sums of up to 256 of them are exact,
    and so is everything that is added in float64.  n particles at one place
    give n times the term, to the last bit."""
    import torch
    x = np.linspace(0.0, 1.0, 4096).astype(F32)
    z = np.zeros(1, F32)

    def sums(count):
        p = torch.tensor([[0.0, 0.0, 0.0]], device="cuda").repeat(count, 1)
        return KDEEstimator(p, bandwidth=0.5)._grid_sum(p, (x, z, z)).cpu().numpy().reshape(-1)

    term = sums(1)
    bits = term.astype(F32).view(np.uint32)
    assert np.array_equal(term.astype(F32).astype(np.float64), term)
    short = (bits & 0x1FF) == 0x100
    assert short.any()
    assert np.array_equal(sums(n)[short], n * term[short])


def _clouds(n, rng):
    return np.concatenate([rng.random((n, 3)), 0.5 + 0.02 * rng.normal(size=(n, 3))]).astype(F32)


@pytest.mark.parametrize("cutoff", [5.0, 6.0])
@pytest.mark.parametrize("n", [1, 20_000])
def test_terms_within_the_cutoff_along_each_axis_are_summed(cutoff, n):
    """One particle near the box's corner, alone within the cutoff of a grid point:
    its term, exp(-3 c^2 / 2) for a share c of the cutoff, is there (to the
    fast exponential's 2^-21 of the exponent, 3 (6)^2 / 2).  The others, far
    away, make the cells fine."""
    import torch
    rng = np.random.default_rng(1)
    h = 0.02
    others = 0.8 + 0.2 * rng.random((n, 3))
    for share in (0.7, 0.9, 0.99):
        d = share * cutoff * h * np.array([[1.0, -1.0, 1.0]])
        P = np.concatenate([0.4 + d, others]).astype(F32)
        k = KDEEstimator(torch.from_numpy(P).cuda(), bandwidth=h, cutoff_sigmas=cutoff)
        ax = np.array([0.4], F32)
        got = float(k._grid_sum(k.P, (ax, ax, ax)).cpu().numpy()[0, 0, 0])
        want = np.exp(-0.5 * (((P[0].astype(np.float64) - np.float64(F32(0.4))) / h) ** 2).sum())
        assert abs(got - want) <= 60 * 2.0 ** -21 * want


@pytest.mark.parametrize("cutoff", [0.7, 2.0, 4.5])
@pytest.mark.parametrize("res", [(5, 7, 8), (17, 3, 20)])
def test_short_cutoffs_sum_the_cells_of_half_a_radius(cutoff, res):
    """A cutoff below 5 sigma decides digits: the sum is over the particles of the
    cells of half a radius that meet the tile grown by it, no more and no less."""
    import torch
    from jaxtrace_gb300 import density as D
    P = _clouds(4000, np.random.default_rng(2))
    k = KDEEstimator(torch.from_numpy(P).cuda(), bandwidth=0.05, cutoff_sigmas=cutoff)
    ax = [np.linspace(0.05, 0.9, r).astype(F32) for r in res]
    got = k._grid_sum(k.P, ax).cpu().numpy()
    r = F32(cutoff * 0.05)
    lo, hi = P.min(axis=0), P.max(axis=0)
    g = D.CellList(k.P, np.minimum(lo, [a[0] for a in ax]), np.maximum(hi, [a[-1] for a in ax]),
                   float(cutoff * 0.05) / 2, 3).grid
    cell = lambda x, a: np.clip(np.floor((x - F32(g.origin[a])) * F32(g.inv_cell[a])), 0, (1 << g.bits) - 1)  # noqa: E731
    mine = [cell(P[:, a], a) for a in range(3)]
    want = np.zeros(res)
    for i in np.ndindex(*[(n + 7) // 8 for n in res]):
        part = [x[8 * b:8 * b + 8] for x, b in zip(ax, i)]
        take = np.ones(len(P), bool)
        for a in range(3):
            take &= (mine[a] >= cell(part[a][0] - r, a)) & (mine[a] <= cell(part[a][-1] + r, a))
        e = [np.exp(-0.5 * ((part[a].astype(np.float64)[:, None] - P[take, a]) / 0.05) ** 2) for a in range(3)]
        want[tuple(slice(8 * b, 8 * b + 8) for b in i)] = np.einsum("ip,jp,kp->ijk", *e)
    assert np.allclose(got, want, rtol=2e-5)
