"""The stencils' 16x4 tiles of small batches against the larger tiles of a batch of copies that is
past their limit: every cell runs the same expressions on the same values, so Jacobian-vector
products and explicit iterations are bitwise equal -- one cell left over in either direction, a
tile cut in both, the last row a tile of its own (both last tile rows touch the far field),
fewer rows than the halo."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu

LIMIT = {np.float64: 2 * 148, np.float32: 4 * 148}


@pytest.mark.parametrize("ni,nc", [(17, 5), (16, 4), (33, 9), (20, 2), (7, 3), (64, 24), (158, 41), (250, 31)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_small_batch_equals_large(cuda, ni, nc, dtype):
    s = EulerSolver(ring(ni, nc), dtype=dtype, device=cuda)
    copies = LIMIT[dtype] // (-(-ni // 16) * -(-nc // 4)) + 1
    rng = np.random.default_rng(ni * nc)
    V = torch.as_tensor(rng.standard_normal((4, ni, nc)), device=cuda)
    out = []
    for B in (1, copies):
        pl = Plan([s.dgrid] * B, s.freestream(np.full(B, 0.6), np.full(B, 2.0)), s.params(), cuda, tuning=None)
        pl.init_freestream()
        U = pl.get_vec(_lib.VEC_U, 0)
        noise = np.random.default_rng(nc).uniform(-0.02, 0.02, (4, ni, nc))
        U = U * (1 + torch.as_tensor(noise, device=cuda))
        for k in (0, B - 1):
            pl.set_vec(_lib.VEC_U, k, U)
            pl.set_vec(_lib.VEC_V, k, V)
        pl.residual()
        pl.jvp()
        R, JV = pl.get_vec(_lib.VEC_R, B - 1), pl.get_vec(_lib.VEC_JV, B - 1)
        pl.rk_iterate(3)
        out.append((R, JV, pl.get_vec(_lib.VEC_U, 0), pl.get_vec(_lib.VEC_U, B - 1)))
        pl.close()
    assert all(torch.isfinite(x).all() for x in out[0])
    for x, y in zip(*out):
        assert torch.equal(x, y)
