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


@pytest.mark.parametrize("n", [1, 10_000, 10_001, 25_000, 25_001, 80_000, 80_001, 100_000,
                               100_001, 300_000])
def test_either_side_of_every_kernel(vg, n):
    ow = random_world(np.random.default_rng(2))
    dw = vg.DeviceWorld(*ow.dims)
    dw.upload(ow.a)
    origin = (-37, 0, 70)
    cams, dirs = rays(np.random.default_rng(n), n, ow.dims, origin)
    b = Batch(cams, dirs)
    b.run(dw, origin)
    b.check(*po.raycast_batch(ow, cams, dirs, origin)[:2])
    dw.close()


@pytest.mark.parametrize("n", [90_000, 110_000])       # lanes to a ray, regions
@pytest.mark.parametrize("seed", range(6))
def test_worlds_and_windows(vg, seed, n):
    rng = np.random.default_rng(seed)
    ow = random_world(rng)
    if seed % 2:        # boxes alone, with empty space of every size between
        b = ow.a["bricks"]
        occ = np.ascontiguousarray(b["occupancy"])
        few = np.unpackbits(occ.view(np.uint8).reshape(-1, 8), axis=1).sum(1) < 8
        b[few] = np.zeros(1, po.BRICK)[0]
        ow.rebuild()
    dw = vg.DeviceWorld(*ow.dims)
    dw.upload(ow.a)
    origin = (0, 0, 0) if seed == 0 else (int(rng.integers(-9000, 9000)), 0,
                                          int(rng.integers(-9000, 9000)))
    cams, dirs = rays(rng, n, ow.dims, origin)
    b = Batch(cams, dirs)
    b.run(dw, origin)
    assert b.check(*po.raycast_batch(ow, cams, dirs, origin)[:2]) > 1000
    dw.close()


@pytest.mark.parametrize("n", [90_000, 110_000])
def test_step_limit(vg, n):
    """8192 empty voxels along x: walks end after 4096 steps, on either side of
    a block placed at the limit, inside an empty region."""
    dims = (2048, 16, 64)
    ow = po.World(*dims)
    for x in (4094, 4095, 4096, 4097):
        ow.set_voxel(x, 8 + x - 4094, 8, 4)
    ow.rebuild()
    dw = vg.DeviceWorld(*dims)
    dw.upload(ow.a)
    y, x0 = np.meshgrid(np.arange(8, 12) + 0.5, np.arange(0, 4) + 0.5)
    cams = np.stack([x0.ravel(), y.ravel(), np.full(x0.size, 8.5)], 1).astype(np.float32)
    cams = np.tile(cams, (n // len(cams) + 1, 1))[:n]
    dirs = np.tile(np.array([[1.0, 0.0, 0.0]], np.float32), (n, 1))
    b = Batch(cams, dirs)
    b.run(dw)
    want = po.raycast_batch(ow, cams[:16], dirs[:16], (0, 0, 0))[:2]
    b.check(*(np.tile(w, n // 16 + 1)[:n] for w in want))
    dw.close()


@pytest.mark.parametrize("name", ["tile_mask", "chunk_mask", "l4_mask"])
def test_masks_that_do_not_hold(vg, name):
    """raycast() reads bricks alone: uploaded masks that miss bricks must not
    hide them, nor after updates of some bricks; generated masks hold again."""
    rng = np.random.default_rng(3)
    ow = random_world(rng)
    a = {k: v.copy() for k, v in ow.a.items()}
    a[name][:] = 0
    dw = vg.DeviceWorld(*ow.dims)
    dw.upload(a)
    cams, dirs = rays(rng, 110_000, ow.dims)
    b = Batch(cams, dirs)
    b.run(dw)
    assert b.check(*po.raycast_batch(ow, cams, dirs, (0, 0, 0))[:2]) > 1000
    idx = np.arange(0, len(ow.a["bricks"]), 97, dtype=np.uint32)
    dw.apply_dirty(idx, ow.a["bricks"][idx])
    b.run(dw)
    b.check(*po.raycast_batch(ow, cams, dirs, (0, 0, 0))[:2])
    dw.generate(vg.TerrainParams(seed=9))
    made = po.World(*ow.dims, arrays=dw.download())
    b.run(dw)
    b.check(*po.raycast_batch(made, cams, dirs, (0, 0, 0))[:2])
    dw.close()


def test_host_batches_on_threads(vg):
    """Batches of several sizes at once on two worlds, each from its own thread,
    single picks between them: every result is the ray's own."""
    import threading
    rng = np.random.default_rng(7)
    worlds = []
    for seed in (4, 5):
        ow = random_world(np.random.default_rng(seed))
        dw = vg.DeviceWorld(*ow.dims)
        dw.upload(ow.a)
        worlds.append((ow, dw))
    jobs, wrong = [], []
    for k, n in enumerate((150_001, 40_000, 12_289, 100, 150_001, 1)):
        ow, dw = worlds[k % 2]
        cams, dirs = rays(rng, n, ow.dims)
        jobs.append((dw, cams, dirs, *po.raycast_batch(ow, cams, dirs, (0, 0, 0))[:2]))

    def work(job):
        dw, cams, dirs, want, want_hit = job
        for _ in range(6):
            hits, found = vg.raycast_batch(dw, cams, dirs)
            sel = want_hit != 0
            if not (np.array_equal(found, want_hit)
                    and np.array_equal(hits["voxel"][sel], want["voxel"][sel])
                    and np.array_equal(hits["normal"][sel], want["normal"][sel])):
                wrong.append(len(cams))
            one = vg.raycast(cams[0], dirs[0], dw)
            if (one is not None) != bool(want_hit[0]):
                wrong.append("single")

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for _, dw in worlds:
        dw.close()
