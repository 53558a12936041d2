"""Implicit residual smoothing in one kernel against the oracle's FFT and Thomas solve, at the edges
of its shapes: rings the Green's function's reach covers whole (ni <= 71) and the first that it
does not, columns that fill no CTA, two rows, and lines too long for its shared memory.

Tolerances, of the largest entry: FP64 1e-12 (as test_smoothing_vs_fft); FP32 the rounding of
at most 72 products of positive weights that add up to one and of a diagonally dominant
solve, 72 eps + 4 eps < 5e-6."""
import numpy as np
import pytest
import torch

from aero2d_b200.euler import EulerSolver
from oracle.euler_oracle import EulerModel
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nc", [(20, 2), (33, 9), (64, 24), (71, 5), (72, 5), (73, 33), (158, 41), (256, 64), (100, 230)])
@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-12), (np.float32, 5e-6)])
def test_smoothing_shapes(cuda, ni, nc, dtype, tol):
    g = ring(ni, nc)
    R = np.random.default_rng(ni + nc).standard_normal((4, ni, nc))
    Ro = EulerModel(g.x, g.y).smooth(R)
    Rs = EulerSolver(g, dtype=dtype, device=cuda).smooth(torch.as_tensor(R)).cpu().numpy()
    assert np.max(np.abs(Rs - Ro)) / np.max(np.abs(Ro)) < tol
