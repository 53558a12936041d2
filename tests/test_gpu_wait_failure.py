"""The failure word that a plan's kernels set when one of their bounded waits runs out: read with the live
count and reported as what it is (the sweeps, the factors and the Arnoldi step all set it).  Set here
from the host; no wait runs out."""
import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

pytestmark = pytest.mark.gpu


def test_failure_word(cuda):
    sv = EulerSolver(ring(64, 12), dtype=np.float32, device=cuda)
    B = 5
    w = sv.freestream(np.linspace(0.4, 0.6, B), np.linspace(0.0, 2.0, B))
    pl = Plan([sv.dgrid] * B, w, sv.params(gmres_restart=2), cuda, tuning=None)
    pl.init_freestream()
    words = pl.workspace[: pl.workspace.numel() // 4 * 4].view(torch.int32)
    before = words.clone()
    assert pl.live_count() == B                      # writes the count; the failure word is beside it
    at = (before != words).nonzero().flatten().tolist()
    assert len(at) == 1 and int(words[at[0]]) == B and int(words[at[0] + 1]) == 0
    words[at[0] + 1] = 1
    with pytest.raises(_lib.A2DError, match="bounded wait.*sweeps.*factors.*Arnoldi"):
        pl.live_count()
    with pytest.raises(_lib.A2DError, match="bounded wait"):
        pl.newton_run(1)
    words[at[0] + 1] = 0
    assert pl.live_count() == B
