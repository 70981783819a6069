"""Pick batches over device arrays (vx_raycast_batch) against the oracle's flat
walk: the kernels that large batches take."""
import ctypes as C

import numpy as np
import pytest

from oracle import pyoracle as po
from scenes import random_world

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vg():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    import voxelg_b200
    return voxelg_b200


class Batch:
    """Rays and results on the device."""

    def __init__(self, cams, dirs):
        import torch
        self.n = len(cams)
        self.cams, self.dirs = (torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
                                for a in (cams, dirs))
        self.out = torch.zeros(self.n * 24, dtype=torch.uint8, device="cuda")
        self.hit = torch.full((self.n,), -1, dtype=torch.int32, device="cuda")

    def run(self, dw, origin=(0, 0, 0)):
        import torch
        from voxelg_b200 import _lib as L
        ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        L.check(L.load().vx_raycast_batch(
            dw.handle, L.i3(origin), ptr(self.cams), ptr(self.dirs), self.n, ptr(self.out),
            ptr(self.hit), C.c_void_p(torch.cuda.current_stream().cuda_stream)))

    def check(self, want, want_hit):
        import torch
        from voxelg_b200 import _lib as L
        torch.cuda.synchronize()
        hits, found = self.out.cpu().numpy().view(L.PICK_DTYPE), self.hit.cpu().numpy()
        assert np.array_equal(found, want_hit)
        sel = found != 0
        for f in ("voxel", "normal"):
            assert np.array_equal(hits[f][sel], want[f][sel])
        return int(sel.sum())


def rays(rng, n, dims, origin=(0, 0, 0)):
    """Random rays, axis-parallel, diagonal and zero directions among them, half
    of the origins on cell planes, some outside the window."""
    size = np.array(dims) * 4
    cams = rng.uniform(-8, size + 8, (n, 3))
    cell = 2.0 ** rng.integers(2, 9, (n, 1))
    snap = (rng.random((n, 3)) < 0.5) & (rng.random((n, 1)) < 0.5)
    cams = np.where(snap, np.round(cams / cell) * cell, cams)
    dirs = rng.normal(size=(n, 3))
    axis = rng.random(n) < 0.2
    dirs[axis] = np.round(dirs[axis])
    tiny = rng.random((n, 3)) < 0.02
    dirs[tiny] *= 1e-42                      # denormal components
    return (cams + origin).astype(np.float32), dirs.astype(np.float32)


def test_captured_batch_meets_masks_that_do_not_hold(vg):
    """A batch captured while the masks held, replayed over uploads whose masks
    miss bricks, and again over one whose masks hold."""
    import torch
    rng = np.random.default_rng(5)
    ow = random_world(rng)
    cams, dirs = rays(rng, 120_001, ow.dims)
    want = po.raycast_batch(ow, cams, dirs, (0, 0, 0))[:2]
    dw = vg.DeviceWorld(*ow.dims)
    dw.upload(ow.a)
    b = Batch(cams, dirs)
    b.run(dw)
    assert b.check(*want) > 1000
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        b.run(dw)
    for name in ("tile_mask", "chunk_mask", "l4_mask"):
        a = {k: v.copy() for k, v in ow.a.items()}
        a[name][:] = 0
        for arrays in (a, ow.a):
            dw.upload(arrays)
            b.hit.fill_(-1)
            graph.replay()
            b.check(*want)
    del graph
    dw.close()
