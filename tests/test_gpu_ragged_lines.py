"""Which kernels apply the preconditioner in ragged batches, and that every
choice gives the per-sweep kernels' bits: several classes of few cases run the per-sweep kernels
together, a large class keeps its one launch beside a case that has none, and long lines in more waves
of clusters than pay run the per-sweep kernels."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu

BATCHES = {   # shapes, one launch for some, per-sweep kernels for some (mixed; FP64; None: a tie)
    "six classes": ([(32 * g, 24) for g in range(4, 10)], (False, True), (False, True)),
    "five sizes": ([(96, 24), (128, 32), (192, 48), (256, 64), (384, 96)] * 2, (False, True), None),
    "two classes": ([(128, 24), (256, 24)], (True, False), (True, False)),
    "a class beside a long ring": ([(544, 6)] + [(256, 64)] * 12, (True, True), (True, True)),
    "the same groups, one past the rows": ([(128, 400)] + [(128, 24)] * 2, (False, True), (False, True)),
    "long lines, many waves": ([(384, 150)] * 16, (False, True), (False, True)),
    "uniform": ([(128, 48)] * 3, (True, False), (True, False)),
}


@pytest.mark.parametrize("name", list(BATCHES))
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_choice(cuda, name, dtype):
    shapes, mixed, fp64 = BATCHES[name]
    solvers = {s: EulerSolver(ring(*s), dtype=dtype, device=cuda) for s in set(shapes)}
    B = len(shapes)
    w = solvers[shapes[0]].freestream(np.linspace(0.4, 0.6, B), np.linspace(0.0, 2.0, B))
    out = []
    rng = np.random.default_rng(B)
    V = [torch.as_tensor(rng.standard_normal((4, *s)), device=cuda) for s in shapes]
    for variant in (("halves" if dtype == np.float32 else "lanes"), "pairs"):
        pl = Plan([solvers[s].dgrid for s in shapes], w, solvers[shapes[0]].params(gmres_restart=2), cuda,
                  tuning=("32x8", variant))
        pl.init_freestream()
        pl.precond_setup()
        for k in range(B):
            pl.set_vec(_lib.VEC_V, k, V[k])
        pl.precond_apply()
        out.append([pl.get_vec(_lib.VEC_JV, k) for k in range(B)])
        want = mixed if dtype == np.float32 else fp64
        if want is not None:
            assert tuple(n in pl.paths() for n in ("lines", "sweeps")) == want
        pl.close()
    assert all(torch.equal(a, b) for a, b in zip(*out))
