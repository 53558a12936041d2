"""A case's explicit iteration does not depend on the cases beside it: alone, and beside one whose lines
are too long for the smoothing's fused kernel, to the bit (an iteration that diverges, as an
unsmoothed one on such a line does, to the same NaN); and the short cases keep that kernel."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu

SHAPES = [(64, 24), (100, 460), (100, 30)]


def iterate(cuda, dtype, which, irs_eps=0.6):
    solvers = [EulerSolver(ring(*SHAPES[k]), dtype=dtype, irs_eps=irs_eps, device=cuda) for k in which]
    w = solvers[0].freestream(np.array([0.4, 0.5, 0.6])[which], np.array([0.0, 1.0, 2.0])[which])
    pl = Plan([s.dgrid for s in solvers], w, solvers[0].params(), cuda, tuning=None)
    pl.init_freestream()
    pl.set_circulation(0.05)
    res = pl.rk_iterate(5)
    out = [(pl.get_vec(_lib.VEC_U, q), res[q]) for q in range(len(which))]
    for q, k in enumerate(which):   # one field smoothed by itself too
        R = np.random.default_rng(k).standard_normal((4, *SHAPES[k]))
        pl.set_vec(_lib.VEC_R, q, torch.as_tensor(R, device=cuda))
    pl.smooth()
    return [(U, r, pl.get_vec(_lib.VEC_R, q)) for q, (U, r) in enumerate(out)]


@pytest.mark.parametrize("irs_eps", [0.6, 0.0])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_alone_and_beside_a_long_line(cuda, dtype, irs_eps):
    together = iterate(cuda, dtype, [0, 1, 2], irs_eps)
    for k in range(len(SHAPES)):
        alone, = iterate(cuda, dtype, [k], irs_eps)
        for a, b in zip(alone, together[k]):
            assert torch.equal(a.view(torch.int64), b.view(torch.int64)), SHAPES[k]


def test_short_cases_keep_the_fused_kernel(cuda):
    solvers = [EulerSolver(ring(*s), dtype=np.float64, device=cuda) for s in SHAPES]
    w = solvers[0].freestream(np.array([0.4, 0.5, 0.6]), np.array([0.0, 1.0, 2.0]))
    pl = Plan([s.dgrid for s in solvers], w, solvers[0].params(), cuda, tuning=None)
    assert {"smooth", "smooth_rows"} <= pl.paths()
    pl.close()
    pl = Plan([solvers[0].dgrid], w[:1], solvers[0].params(), cuda, tuning=None)
    assert "smooth" in pl.paths() and "smooth_rows" not in pl.paths()
