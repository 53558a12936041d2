"""The smoothing at coefficients whose Green's function ends within a rounding of an integer reach, where
a logarithm that rounds the other way moves the reach by one: the shared memory is sized by the
same reach that the kernels run with.  Against the sum over the Green's function's closed form (whose
lam cancels at small coefficients, so the FFT's solution is no reference there) and the oracle's
Thomas solve, 1e-12 of the largest entry as the smoothing's other tests in FP64; the term in
question is 1e-18 of it."""
import numpy as np
import pytest
import torch

from aero2d_b200.euler import EulerSolver
from oracle.euler_oracle import thomas
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu


def smoothed(R, e):
    ni, nc = R.shape[1:]
    lam = ((1 + 2 * e) - np.sqrt(1 + 4 * e)) / (2 * e)
    g0 = 1 / (e * (1 / lam - lam))
    m = np.arange(ni // 2 + 1)
    g = g0 * (lam ** m + lam ** (ni - m)) / (1 - lam ** ni)
    S = g[0] * R
    for d in range(1, ni):
        S = S + g[min(d, ni - d)] * np.roll(R, d, axis=1)
    dl, d, du = np.full(nc, -e), np.full(nc, 1 + 2 * e), np.full(nc, -e)
    dl[0] = du[-1] = 0.0
    d[0] = d[-1] = 1 + e
    return thomas(dl, d, du, S)


@pytest.mark.parametrize("reach", [7, 8, 12, 16, 35, 36, 40])
def test_reach_at_an_integer(cuda, reach):
    lam = 10.0 ** (-18.0 / reach)
    mid = lam / (1.0 - lam) ** 2           # lam of this coefficient: lam^reach = 1e-18
    ni, nc = 100, 13
    g = ring(ni, nc)
    R = np.random.default_rng(reach).standard_normal((4, ni, nc))
    for ulps in (-4, -1, 0, 1, 4):
        e = mid + ulps * np.spacing(mid)
        Ro = smoothed(R, e)
        Rs = EulerSolver(g, dtype=np.float64, irs_eps=e, device=cuda).smooth(torch.as_tensor(R)).cpu().numpy()
        assert np.max(np.abs(Rs - Ro)) / np.max(np.abs(Ro)) < 1e-12


@pytest.mark.parametrize("ni", [4, 8, 9, 10, 11, 14])
@pytest.mark.parametrize("e", [1e-3, 1e-6])
def test_small_rings_shorter_than_a_block_of_columns(cuda, ni, e):
    """Rings that a CTA's 32 columns go round several times, with a reach that does not cover them."""
    nc = 5
    R = np.random.default_rng(ni).standard_normal((4, ni, nc))
    Ro = smoothed(R, e)
    Rs = EulerSolver(ring(ni, nc), dtype=np.float64, irs_eps=e, device=cuda).smooth(torch.as_tensor(R)).cpu().numpy()
    assert np.max(np.abs(Rs - Ro)) / np.max(np.abs(Ro)) < 1e-12
