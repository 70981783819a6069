"""Updates of bricks either side of the sizes where the kernels that re-derive
the parent words change, repeated bricks among them: every array equals the
oracle's rebuild."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_edit_update import random_bricks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [383, 384, 385, 19_999, 20_000, 20_001, 70_001])
def test_update_equals_rebuild(n):
    import torch
    import voxelg_b200 as vg
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    rng = np.random.default_rng(n)
    dims = (64, 16, 128)
    nb = dims[0] * dims[1] * dims[2]
    ow = po.World(*dims)
    dw = vg.DeviceWorld(*dims)
    for turn in range(2):
        idx = rng.integers(0, nb // (1 + turn * 7), n).astype(np.uint32)
        b = random_bricks(rng, n)
        if turn:
            b[: n // 2] = np.zeros(1, po.BRICK)[0]
        dw.apply_dirty(idx, b)
        last = dict(zip(idx.tolist(), range(n)))          # the last entry of a brick wins
        ow.a["bricks"][list(last)] = b[list(last.values())]
        ow.rebuild()
        got = dw.download()
        for k in po.World.NAMES:
            assert np.array_equal(got[k].view(np.uint8), ow.a[k].view(np.uint8)), (turn, k)
    dw.close()
