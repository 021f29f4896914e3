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
