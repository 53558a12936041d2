"""Plan calls under stream capture: a captured call must leave no host state behind that a call made
before the graph's first replay, or after a dropped capture, takes for work done."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu


def fresh(cuda, dtype):
    sv = EulerSolver(ring(96, 24), dtype=dtype, device=cuda)
    pl = Plan([sv.dgrid], sv.freestream(np.array([0.5]), np.array([1.5])), sv.params(), cuda, tuning=None)
    pl.init_freestream()
    pl.set_circulation(0.1)
    return pl


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_explicit_iteration_captured_first(cuda, dtype):
    """Direct iterations before any replay of a captured one, then the replay: both as without a capture."""
    plain = fresh(cuda, dtype)
    want = []
    for _ in range(2):
        plain.rk_iterate(3)
        want.append(plain.get_vec(_lib.VEC_U, 0))
    pl = fresh(cuda, dtype)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pl.rk_iterate(3)
    pl.rk_iterate(3)
    assert torch.equal(pl.get_vec(_lib.VEC_U, 0), want[0])
    graph.replay()
    assert torch.equal(pl.get_vec(_lib.VEC_U, 0), want[1])
    torch.cuda.synchronize()
    del graph


def test_smoothing_after_a_dropped_capture(cuda):
    R = torch.as_tensor(np.random.default_rng(3).standard_normal((4, 96, 24)), device=cuda)

    def smoothed(pl):
        pl.set_vec(_lib.VEC_R, 0, R)
        pl.smooth()
        return pl.get_vec(_lib.VEC_R, 0)

    want = smoothed(fresh(cuda, np.float64))
    pl = fresh(cuda, np.float64)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pl.smooth()
    del graph
    assert torch.equal(smoothed(pl), want)
