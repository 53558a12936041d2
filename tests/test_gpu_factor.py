"""The line factors at the edges of their kernel's shapes: no row beyond the twist on the far side,
one, fewer rows than helper warps, several rounds of them with one left over; a single partial
line group; and both helper counts, one case alone and a batch of more than 148 line groups.
One application of one sweep, bitwise equal in either batch, in FP64 against the oracle's
block-Thomas solve: these lines amplify a right-hand side up to 240 times, rounding of some
100 operations a row on the way stays below 1e-10 of the largest entry."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from oracle.euler_oracle import EulerModel
from oracle.implicit_oracle import ImplicitModel
from tests.helpers import perturbed_state
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nc", [(20, 2), (33, 3), (7, 5), (64, 13), (40, 17), (31, 44)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_factor_shapes(cuda, ni, nc, dtype):
    g = ring(ni, nc)
    om = EulerModel(g.x, g.y)
    im = ImplicitModel(om, jacobi_sweeps=1)
    w = om.freestream(0.55, 1.0)
    U = perturbed_state(om, w, seed=2, amp=0.01)
    cfl = 37.0
    circ = im.circ(U, w)
    R, W = om.residual(U, w, circ)
    D, Bim, Bip, Bjm, Bjp = im.assemble(U, w, circ, 1.0 / (om.local_dt(W) / om.cfl * cfl))
    fac = im.factor_lines(D, Bjm, Bjp)
    r = np.random.default_rng(9).standard_normal(U.shape)
    xo = im.precond(fac, Bim, Bip, r)
    s = EulerSolver(g, dtype=dtype, device=cuda)
    x = []
    for B in (1, 148 // -(-ni // 32) + 1):
        pl = Plan([s.dgrid] * B, np.tile(w, (B, 1)), s.params(jacobi_sweeps=1), cuda, tuning=None)
        pl.init_freestream()
        for k in {0, B - 1}:
            pl.set_vec(_lib.VEC_U, k, torch.as_tensor(U))
            pl.set_vec(_lib.VEC_V, k, torch.as_tensor(r))
        pl.set_cfl([cfl] * B)
        pl.precond_setup()
        pl.precond_apply()
        x += [pl.get_vec(_lib.VEC_JV, k) for k in (0, B - 1)]
        pl.close()
    assert torch.isfinite(x[0]).all()
    if dtype == np.float64:
        assert np.max(np.abs(x[0].cpu().numpy() - xo)) / np.max(np.abs(xo)) < 1e-10
    assert all(torch.equal(y, x[0]) for y in x[1:])
