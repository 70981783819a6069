"""Picking that skips empty regions (batches) and takes 32 steps a round
(single calls), against the oracle's flat walk: every face and corner of
bricks, tiles, chunks and L4 cells, shifted windows, starts inside solids and
fringe, the 4096-step limit, masks that do not hold for the bricks."""
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


def check(vg, dw, ow, cams, dirs, origin, singles=200):
    hits, found = vg.raycast_batch(dw, cams, dirs, origin)
    want, want_hit, _ = po.raycast_batch(ow, cams, dirs, origin)
    assert np.array_equal(found, want_hit)
    sel = found != 0
    assert np.array_equal(hits["voxel"][sel], want["voxel"][sel])
    assert np.array_equal(hits["normal"][sel], want["normal"][sel])
    for i in np.linspace(0, len(cams) - 1, singles).astype(int):
        h = vg.raycast(cams[i], dirs[i], dw, origin)
        assert (h is not None) == bool(want_hit[i]), i
        if h is not None:
            assert h.voxel == tuple(want["voxel"][i]) and h.normal == tuple(want["normal"][i]), i
    return int(sel.sum())


def rays(rng, n, dims, origin):
    """Random rays with axis-parallel and diagonal directions among them, half
    of the origins on cell planes, some outside the window."""
    size = np.array(dims) * 4
    cams = rng.uniform(-8, size + 8, (n, 3))
    cell = 2.0 ** rng.integers(2, 9, (n, 1))
    snap = rng.random((n, 3)) < 0.5
    cams = np.where(snap & (rng.random((n, 1)) < 0.5), np.round(cams / cell) * cell, cams)
    dirs = rng.normal(size=(n, 3))
    axis = rng.random(n) < 0.2
    dirs[axis] = np.round(dirs[axis])
    return ((cams + origin).astype(np.float32), dirs.astype(np.float32))


@pytest.mark.parametrize("seed", range(6))
def test_random_worlds_and_windows(vg, seed):
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
    # window corners off every cell's grid
    origin = (0, 0, 0) if seed == 0 else (int(rng.integers(-9000, 9000)), 0,
                                          int(rng.integers(-9000, 9000)))
    cams, dirs = rays(rng, 4000, ow.dims, origin)
    assert check(vg, dw, ow, cams, dirs, origin) > 100
    dw.close()


def test_step_limit(vg):
    """8192 empty voxels along x: walks end after 4096 steps, on either side
    of a block placed at the limit."""
    dims = (2048, 16, 64)
    ow = po.World(*dims)
    for x in (4094, 4095, 4096, 4097):
        ow.set_voxel(x, 8 + x - 4094, 8, 4)
    ow.rebuild()
    dw = vg.DeviceWorld(*dims)
    dw.upload(ow.a)
    y, x0 = np.meshgrid(np.arange(8, 12) + 0.5, np.arange(0, 4) + 0.5)
    cams = np.stack([x0.ravel(), y.ravel(), np.full(x0.size, 8.5)], 1).astype(np.float32)
    dirs = np.tile(np.array([[1.0, 0.0, 0.0]], np.float32), (len(cams), 1))
    check(vg, dw, ow, cams, dirs, (0, 0, 0), singles=len(cams))
    dw.close()


def test_masks_that_do_not_hold(vg):
    """raycast() reads bricks alone: uploaded masks that miss bricks must not
    hide them."""
    rng = np.random.default_rng(3)
    ow = random_world(rng)
    cams, dirs = rays(rng, 3000, ow.dims, (0, 0, 0))
    dw = vg.DeviceWorld(*ow.dims)
    for name in ("tile_mask", "chunk_mask", "l4_mask"):
        a = {k: v.copy() for k, v in ow.a.items()}
        a[name][:] = 0
        dw.upload(a)
        assert check(vg, dw, ow, cams, dirs, (0, 0, 0), singles=50) > 100
    dw.close()


@pytest.mark.parametrize("n", [0, 1, 31, 8193, 10001, 25001, 32769, 80001, 100001, 140000])
def test_batch_sizes(vg, n):
    """Either side of the sizes where a batch is cut into chunks and where the
    lanes to a ray change."""
    rng = np.random.default_rng(n)
    ow = random_world(np.random.default_rng(2))
    dw = vg.DeviceWorld(*ow.dims)
    dw.upload(ow.a)
    cams, dirs = rays(rng, n, ow.dims, (-37, 0, 70))
    check(vg, dw, ow, cams, dirs, (-37, 0, 70), singles=min(n, 5))
    dw.close()
