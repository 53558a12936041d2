"""The Gram-Schmidt passes on sizes whose chunks end inside a row (the last chunk short, down to a
few entries), in few chunks (a chunk's rows on CTAs of their own) and in many (a CTA per chunk),
with bases past 32 vectors: a Newton step of one FP64 case against the oracle's, and the
same cases alone and together bitwise the same in FP64 and in mixed precision.

The tolerance of the oracle comparison is that of test_one_newton_step_vs_oracle (the
rounding of a GMRES cycle)."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.implicit import ImplicitEuler
from aero2d_b200.plan import Plan
from oracle.euler_oracle import EulerModel
from oracle.implicit_oracle import ImplicitModel
from tests.helpers import grid, perturbed_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nj,restart", [(33, 18, 1), (33, 25, 33), (41, 26, 40)])
def test_newton_step_vs_oracle(cuda, ns, nj, restart):
    g = grid("0012", ns, nj)
    om = EulerModel(g.x, g.y)
    w = om.freestream(0.5, 2.0)
    U = perturbed_state(om, w, seed=3, amp=0.01)
    Uo, rno, omo, _ = ImplicitModel(om, gmres_restart=restart).step(U, w, 10.0)
    s = ImplicitEuler(EulerSolver(g, dtype=np.float64, device=cuda), gmres_restart=restart)
    Ug, rng, omg = s.step(torch.as_tensor(U), w, None, 10.0)
    assert abs(rng - rno) / rno < 1e-12 and abs(omg - omo) < 1e-8
    dU = Uo - U
    assert np.max(np.abs((Ug.cpu().numpy() - U) - dU)) / np.max(np.abs(dU)) < 1e-7


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_few_and_many_chunks_same_results(cuda, dtype):
    """A case alone (7 chunks, the last of 1408 entries) and among 12 (84 chunks)."""
    base = EulerSolver(grid("2412", 65, 53), dtype=dtype, device=cuda)
    machs, alphas = np.linspace(0.4, 0.7, 12), np.linspace(-2.0, 4.0, 12)
    w = base.freestream(machs, alphas)
    par = ImplicitEuler(base, gmres_restart=36).params(1e-10, 10)
    out = {}
    for ks in (range(12), [7]):
        pl = Plan([base.dgrid] * len(ks), w[list(ks)], par, cuda, tuning=None)
        pl.init_freestream()
        for _ in range(3):
            pl.newton_step()
        out[len(ks)] = (pl.get_vec(_lib.VEC_U, len(ks) - 5 if len(ks) > 1 else 0), pl.scalars()[-5 if len(ks) > 1 else 0])
        pl.close()
    assert torch.isfinite(out[1][0]).all()
    assert torch.equal(out[12][0], out[1][0]) and np.array_equal(out[12][1], out[1][1])
