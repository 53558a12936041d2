"""The line preconditioner's one-launch kernel (a cluster per case) against the per-sweep
kernels, which compute the same arithmetic in the same order: bitwise equal on every edge of
its shapes -- one line in the last group, a single group (a CTA its own neighbour), the largest
cluster, two rows (no far-field rows), packs cut short on either side, all sizes in one ragged
batch -- for one to four sweeps, each application on a right-hand side of its own."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.grid import OGrid
from aero2d_b200.plan import Plan

pytestmark = pytest.mark.gpu

SHAPES = [(128, 32), (96, 24), (80, 42), (33, 9), (20, 2), (64, 3), (512, 17), (7, 5), (250, 64)]


def ring(ni, nc):
    """A ring of cells round a wavy oval: any ni >= 4, nc >= 2."""
    th = -2 * np.pi * np.arange(ni) / ni
    r = 0.5 * 40 ** (np.arange(nc + 1) / nc)
    g = OGrid(0.5 + np.outer(np.cos(th) * (1 + 0.1 * np.cos(3 * th)), r), 0.8 * np.outer(np.sin(th), r))
    return g if g.cell_areas().min() > 0 else OGrid(g.x[::-1].copy(), g.y[::-1].copy())


@pytest.mark.parametrize("sweeps", [1, 2, 3, 4])
@pytest.mark.parametrize("dtype,one", [(np.float64, "lanes"), (np.float32, "halves")])
def test_one_launch_equals_per_sweep(cuda, dtype, one, sweeps):
    solvers = [EulerSolver(ring(*s), dtype=dtype, device=cuda) for s in SHAPES]
    B = len(solvers)
    w = solvers[0].freestream(np.linspace(0.4, 0.7, B), np.linspace(-1.0, 3.0, B))
    pl = Plan([s.dgrid for s in solvers], w, solvers[0].params(jacobi_sweeps=sweeps), cuda, tuning=None)
    pl.init_freestream()
    pl.precond_setup()
    rng = np.random.default_rng(sweeps)

    def apply(variant, V):
        pl.set_tuning("32x8", variant)
        for k in range(B):
            pl.set_vec(_lib.VEC_V, k, V[k])
        pl.precond_apply()
        return [pl.get_vec(_lib.VEC_JV, k) for k in range(B)]

    for _ in range(3):
        V = [torch.as_tensor(rng.standard_normal((4, s.ni, s.nc)), device=cuda) for s in solvers]
        a, b = apply(one, V), apply("pairs", V)
        assert all(torch.isfinite(x).all() for x in a)
        for x, y, s in zip(a, b, SHAPES):
            assert torch.equal(x, y), s
    pl.close()


def test_more_lines_than_a_cluster_takes(cuda):
    """A case of more than 512 lines runs the per-sweep kernels, and the cases beside it too."""
    shapes = [(544, 6), (64, 6)]
    solvers = [EulerSolver(ring(*s), dtype=np.float32, device=cuda) for s in shapes]
    w = solvers[0].freestream(np.array([0.5, 0.6]), np.array([1.0, 2.0]))
    out = {}
    rng = np.random.default_rng(1)
    V = [torch.as_tensor(rng.standard_normal((4, s.ni, s.nc)), device=cuda) for s in solvers]
    for v in ("halves", "rows"):
        pl = Plan([s.dgrid for s in solvers], w, solvers[0].params(), cuda, tuning=("32x8", v))
        pl.init_freestream()
        pl.precond_setup()
        for k in range(2):
            pl.set_vec(_lib.VEC_V, k, V[k])
        pl.precond_apply()
        out[v] = [pl.get_vec(_lib.VEC_JV, k) for k in range(2)]
        pl.close()
    assert all(torch.equal(x, y) for x, y in zip(out["halves"], out["rows"]))
