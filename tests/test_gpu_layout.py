"""Cell vectors in and out of a plan: exact for every case of a ragged batch (cells that fill no
tile, one row of a tile, one column), one case at a time and all at once, with the neighbours
of a case untouched."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu


def plan(shapes, cuda):
    solvers = [EulerSolver(ring(*s), dtype=np.float64, device=cuda) for s in shapes]
    B = len(shapes)
    return Plan([s.dgrid for s in solvers], solvers[0].freestream(np.full(B, 0.5), np.full(B, 1.0)),
                solvers[0].params(), cuda, tuning=None)


def test_ragged_one_by_one(cuda):
    shapes = [(33, 9), (7, 3), (64, 24), (20, 2), (31, 17), (158, 41)]
    pl = plan(shapes, cuda)
    rng = np.random.default_rng(3)
    V = [torch.as_tensor(rng.uniform(0.5, 1.5, (4, *s)), device=cuda) for s in shapes]
    for k in (3, 0, 5, 1, 4, 2):
        pl.set_vec(_lib.VEC_V, k, V[k])
    for k, v in enumerate(V):
        assert torch.equal(pl.get_vec(_lib.VEC_V, k), v)
        w = pl.get_prim(_lib.VEC_V, k)
        assert torch.equal(w[0], v[0])
        assert torch.allclose(w[1], v[1] / v[0], rtol=1e-15, atol=0)
        assert torch.allclose(w[3], 0.4 * (v[3] - 0.5 * (v[1] ** 2 + v[2] ** 2) / v[0]), rtol=0, atol=4e-15)
    with pytest.raises(RuntimeError):
        pl.get_batch(_lib.VEC_V)
    pl.close()


@pytest.mark.parametrize("ni,nc", [(33, 9), (20, 2), (64, 24), (7, 17)])
def test_batch(cuda, ni, nc):
    pl = plan([(ni, nc)] * 3, cuda)
    V = torch.as_tensor(np.random.default_rng(ni).standard_normal((4, 4, ni, nc)), device=cuda)
    pl.set_batch(_lib.VEC_V, V[:3])
    assert torch.equal(pl.get_batch(_lib.VEC_V), V[:3])
    assert all(torch.equal(pl.get_vec(_lib.VEC_V, k), V[k]) for k in range(3))
    strided = V.transpose(2, 3).contiguous().transpose(2, 3)    # the same values, other strides
    for other in (V, strided[:3], V[:3].cpu(), V[:3].float(), [V[k] for k in range(3)]):
        pl.set_batch(_lib.VEC_DU, torch.zeros_like(V[:3]))
        pl.set_batch(_lib.VEC_DU, other)
        want = torch.stack([torch.as_tensor(other[k]).to(cuda, torch.float64) for k in range(3)])
        assert torch.equal(pl.get_batch(_lib.VEC_DU), want)
    with pytest.raises(ValueError):
        pl.set_batch(_lib.VEC_V, V[:3, :, :, :-1])
    with pytest.raises(IndexError):
        pl.set_batch(_lib.VEC_V, V[:2])
    pl.close()
