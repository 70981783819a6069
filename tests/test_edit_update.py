"""The dirty-brick update around the size where its launch form changes, and
the tile projection at mask-word and row edges, against the oracle."""
import math

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vg():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    import voxelg_b200
    return voxelg_b200


def random_bricks(rng, n):
    """n bricks: random, empty, full of one material, full of two."""
    b = np.zeros(n, po.BRICK)
    kind = rng.integers(0, 4, n)
    mats = rng.integers(1, 5, (n, 64)).astype(np.uint8)
    solid = rng.random((n, 64)) < 0.5
    solid[kind == 1] = False
    solid[kind >= 2] = True
    mats[kind == 2] = mats[kind == 2, :1]
    b["materials"] = np.where(solid, mats, 0)
    b["occupancy"] = np.packbits(solid, axis=1, bitorder="little").view(np.uint64)[:, 0]
    return b


@pytest.mark.parametrize("n", [1, 2, 33, 128, 129, 1023, 1024, 1025, 2500])
def test_dirty_update_equals_rebuild(vg, n):
    """Uniform tiles, emptied tiles, chunks and L4 cells, repeated bricks:
    every array equals the oracle's rebuild after each of two updates."""
    rng = np.random.default_rng(n)
    dims = (64, 16, 128)
    nb = dims[0] * dims[1] * dims[2]
    ow = po.World(*dims)
    dw = vg.DeviceWorld(*dims)
    for turn in range(2):
        # half of the entries fill whole tiles, the rest fall in a small range
        idx = rng.integers(0, nb // 8, n)
        tile = rng.integers(0, dims[0] // 4, n // 64 + 1)[np.arange(n // 2) // 64]
        c = np.arange(n // 2) % 64
        idx[:n // 2] = tile * 4 + (c & 3) + (c >> 4) * 64 + ((c >> 2) & 3) * 64 * 16
        idx = idx.astype(np.uint32)
        b = random_bricks(rng, n)
        b[:n // 2] = b[n // 2] if turn == 0 else np.zeros(1, po.BRICK)[0]
        dw.apply_dirty(idx, b)
        for i in range(n):
            ow.a["bricks"][idx[i]] = b[i]
        ow.rebuild()
        got = dw.download()
        for k in po.World.NAMES:
            assert np.array_equal(got[k].view(np.uint8), ow.a[k].view(np.uint8)), (turn, k)
    dw.close()


@pytest.mark.parametrize("size", [(1, 1), (8, 300), (255, 97), (256, 64), (257, 65), (1920, 1080)])
def test_projection_fills_the_same_tiles(vg, size):
    """Single tiles, wide and tall rectangles and bricks across the camera
    plane (the whole screen) on tile rows of 1 to 240 tiles."""
    import torch
    W, H = size
    dims = (64, 16, 64)
    ow = po.World(*dims)
    dw = vg.DeviceWorld(*dims)
    rng = np.random.default_rng(W)
    cam = vg.camera_from_pose((128.0, 32.0, 128.0), 0.4, math.radians(-15.0), math.radians(70.0),
                              W, H)
    near = np.array([(x >> 2) + (y >> 2) * 64 + (z >> 2) * 64 * 16
                     for x, y, z in rng.integers((120, 24, 120), (145, 40, 145), (24, 3))])
    far = rng.integers(0, 64 * 16 * 64, 24)
    groups = [[int(i)] for i in np.concatenate([near, far])] + [near.tolist(), far.tolist()]
    for g in groups:
        mask = torch.zeros(vg.tile_mask_words(W, H), dtype=torch.int32, device="cuda")
        vg.project_dirty(dw, cam, np.array(g, np.uint32), mask)
        assert np.array_equal(mask.cpu().numpy().view(np.uint32), po.project_dirty(ow, cam, g)), g
    dw.close()
