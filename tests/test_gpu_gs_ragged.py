"""One-launch Arnoldi steps of a ragged batch: cases of one to six chunks in clusters of the largest one's
size, so that most CTAs of the small ones have no row.  Each case takes the steps that it takes alone,
to the bit."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu

SHAPES = [(32, 8), (128, 48), (40, 13), (96, 24), (64, 33), (33, 31)]   # 1, 6, 1, 3, 3, 1 chunks


def test_ragged_equals_alone(cuda):
    solvers = [EulerSolver(ring(*s), dtype=np.float32, device=cuda) for s in SHAPES]
    w = solvers[0].freestream(np.linspace(0.4, 0.6, len(SHAPES)), np.linspace(-1.0, 2.0, len(SHAPES)))

    def run(which):
        pl = Plan([solvers[k].dgrid for k in which], w[which], solvers[0].params(gmres_restart=20), cuda, tuning=None)
        assert "arnoldi" in pl.paths()
        pl.init_freestream()
        for _ in range(3):
            pl.newton_step()
        return [pl.get_vec(_lib.VEC_U, q) for q in range(len(which))], pl.scalars()

    U, sc = run(list(range(len(SHAPES))))
    for k in range(len(SHAPES)):
        (u,), s = run([k])
        assert torch.isfinite(u).all() and torch.equal(u, U[k]), SHAPES[k]
        assert np.array_equal(s[0], sc[k], equal_nan=True)
