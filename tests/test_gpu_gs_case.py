"""Arnoldi steps in one launch, a cluster per case, against the three passes, which the same cases take
beside one too large for it: bitwise equal after two Newton steps.  Fewer rows than CTAs, a last
chunk with empty rows and with part of one, five rows to a CTA, cycles longer than the shared
memory holds vectors for (the later steps by passes), and two cases at once."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.implicit import ImplicitEuler
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nc,restart", [(16, 4, 5), (20, 2, 12), (33, 9, 30), (64, 24, 40), (96, 41, 64), (160, 64, 40)])
def test_one_launch_equals_passes(cuda, ni, nc, restart):
    small, large = (EulerSolver(ring(*s), dtype=np.float32, device=cuda) for s in ((ni, nc), (256, 64)))
    par = ImplicitEuler(small, gmres_restart=restart).params(1e-10, 10)
    w = small.freestream(np.array([0.45, 0.6, 0.5]), np.array([1.0, 3.0, 2.0]))
    out = []
    for grids in ([small.dgrid] * 2, [small.dgrid] * 2 + [large.dgrid]):
        pl = Plan(grids, w[:len(grids)], par, cuda, tuning=None)
        pl.init_freestream()
        for _ in range(2):
            pl.newton_step()
        out.append([pl.get_vec(_lib.VEC_DU, k) for k in range(2)] + [torch.as_tensor(pl.scalars()[:2])])
        pl.close()
    assert all(torch.isfinite(x).all() for x in out[0][:2])
    assert all(torch.equal(x, y) for x, y in zip(*out))
