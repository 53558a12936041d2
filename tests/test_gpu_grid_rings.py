"""The device grid march at the edges of its windows."""
import numpy as np
import pytest
import torch

from aero2d_b200.grid import ogrid
from aero2d_b200.gridgen import ogrid_batch
from aero2d_b200.plan import DeviceGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni", [24, 44, 45, 64, 88, 90, 130, 500, 1024])
def test_ring_sizes(cuda, ni):
    """Rings that a warp's window wraps round more than once, that end on a warp's last point or one
    past it, and the largest, against the host's smoothing: layers 0 .. nj-2 bitwise, the
    metrics of every grid of the batch those of its own nodes."""
    class Blob:
        def __init__(self, k):
            t = 2 * np.pi * np.arange(ni + 1) / ni
            r = 0.5 + 0.02 * np.cos(2 * t + k)
            self.c = np.stack([0.5 + r * np.cos(t), r * np.sin(t)], axis=1)
            self.c[-1] = self.c[0]

        def coords(self):
            return self.c

    blobs = [Blob(k) for k in range(3)]
    grids = ogrid_batch(blobs, nj=9, ds0=2e-2, radius=4.0, device=cuda)
    for b, g in zip(blobs, grids):
        h = ogrid(b, nj=9, ds0=2e-2, radius=4.0)
        x, y = g.x.cpu().numpy(), g.y.cpu().numpy()
        assert np.array_equal(x[:, :-1], h.x[:, :-1]) and np.array_equal(y[:, :-1], h.y[:, :-1])
        assert np.max(np.abs(x[:, -1] - h.x[:, -1])) < 1e-13 and np.max(np.abs(y[:, -1] - h.y[:, -1])) < 1e-13
        one = DeviceGrid(nodes=(g.x, g.y))
        n64 = 8 * (5 * ni * g.nc + 6 * ni)      # the FP64 part; padding, which nothing writes, follows
        n32 = 4 * (5 * ni * g.nc + 4 * ni)      # the FP32 part, at the end
        size = one.metrics.numel()
        assert torch.equal(one.metrics[:n64], g.metrics[:n64])
        assert torch.equal(one.metrics[size - n32:], g.metrics[size - n32:size])
