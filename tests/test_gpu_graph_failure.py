"""A Newton step whose graph cannot be made: instantiation is not permitted while the same thread
captures another stream.  A step either is made and counted or is refused with nothing run, and the
steps after the capture go on as without it.  In a process of its own, since the capture is
invalidated by the attempt."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import numpy as np, torch
from aero2d_b200 import _lib
from aero2d_b200.euler import EulerSolver
from aero2d_b200.plan import Plan
from tests.test_gpu_lines import ring

cuda = torch.device("cuda", 0)
sv = EulerSolver(ring(96, 24), dtype=np.float32, device=cuda)

def fresh():
    pl = Plan([sv.dgrid], sv.freestream(np.array([0.5]), np.array([1.5])), sv.params(), cuda, tuning=None)
    pl.init_freestream()
    torch.cuda.synchronize()
    return pl

def state(pl):
    U = pl.get_vec(_lib.VEC_U, 0)
    torch.cuda.synchronize()
    return U

plain = fresh()
want = []
for _ in range(2):
    plain.newton_step()
    want.append(state(plain))

pl = fresh()
other, x = torch.cuda.Stream(), torch.zeros(8, device=cuda)
graph, refused, invalid = torch.cuda.CUDAGraph(), None, False
torch.cuda.synchronize()
try:
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        x.add_(1)
        with torch.cuda.stream(other):
            pl.newton_step()
            try:
                pl.newton_step()
            except _lib.A2DError as e:
                refused = str(e)
except Exception:
    invalid = True
assert refused is not None and "graph" in refused, refused
assert invalid
torch.cuda.synchronize()
assert pl.stats()[1] == 1 and torch.equal(state(pl), want[0])
pl.newton_step()
assert pl.stats()[1] == 2 and torch.equal(state(pl), want[1])
print("done")
"""


def test_no_error_follows_a_step(cuda):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=Path(__file__).resolve().parents[1], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
