"""The metrics of a batch of grids: one launch per 128 grids, each blob the one that its grid makes alone and
in memory of its own, so that a grid kept from a batch keeps no other's."""
import ctypes as C

import numpy as np
import pytest
import torch

from aero2d_b200 import _lib
from aero2d_b200.geometry import naca4
from aero2d_b200.gridgen import ogrid_batch
from aero2d_b200.plan import DeviceGrid, _ptr

pytestmark = pytest.mark.gpu


def blob_bytes(ni, nj):
    n = C.c_size_t()
    _lib.check(_lib.load().a2d_metrics_bytes(ni, nj, C.byref(n)))
    return n.value


def test_a_kept_grid_keeps_its_own_metrics(cuda):
    grids = ogrid_batch([naca4(c, 33) for c in ("0012", "2412", "4412")], nj=17, device=cuda)
    for g in grids:
        assert g.metrics.untyped_storage().nbytes() == blob_bytes(g.ni, g.nj)
        assert torch.equal(g.metrics, DeviceGrid(nodes=(g.x, g.y)).metrics)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 300])
def test_more_grids_than_a_launch_takes(cuda, n):
    ni, nj = 9, 4
    rng = np.random.default_rng(n)
    th = -2 * np.pi * np.arange(ni) / ni
    r = 1.0 + np.arange(nj)[None, :] + 0.1 * rng.uniform(size=(n, 1, nj))
    x = torch.as_tensor(np.cos(th)[None, :, None] * r, device=cuda).contiguous()
    y = torch.as_tensor(np.sin(th)[None, :, None] * r, device=cuda).contiguous()
    size = blob_bytes(ni, nj)
    blobs = [torch.zeros(size, dtype=torch.uint8, device=cuda) for _ in range(n)]
    stride = -(-size // 256) * 256
    one = torch.zeros((n, stride), dtype=torch.uint8, device=cuda)
    lib, s = _lib.load(), torch.cuda.current_stream().cuda_stream
    _lib.check(lib.a2d_metrics_build_each(n, ni, nj, _ptr(x), _ptr(y), (C.c_void_p * n)(*map(_ptr, blobs)), s))
    _lib.check(lib.a2d_metrics_build_batch(n, ni, nj, _ptr(x), _ptr(y), _ptr(one), stride, s))
    for k in range(n):
        alone = torch.zeros(size, dtype=torch.uint8, device=cuda)
        _lib.check(lib.a2d_metrics_build(ni, nj, _ptr(x[k]), _ptr(y[k]), _ptr(alone), s))
        assert torch.equal(blobs[k], alone) and torch.equal(one[k, :size], alone)
