"""The queue's packets of 32 rays, sorted and not, over mixed kinds: below, at
and beyond a packet for every warp that a B200 holds, and past the sizes where
the sort's key is shortened.  Every record equals vx_trace's."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    import voxelg_b200 as vg
    cfg = vg.CONFIGS["c1"]
    dw = vg.DeviceWorld(*cfg.bricks)
    dw.generate(cfg.terrain)
    yield vg, dw
    dw.close()


@pytest.mark.parametrize("sort", [0, 1])
@pytest.mark.parametrize("n", [33, 75_777, 113_664, 113_665, 524_288, 524_289, 1_100_001])
def test_mixed_kinds(gpu, n, sort):
    import torch
    import voxelg_b200.queue as q
    vg, dw = gpu
    rng = np.random.default_rng(n)
    rays = np.zeros(n, po.RAY)
    rays["org"] = rng.uniform([-20, 20, -20], [532, 240, 532], (n, 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[rng.random((n, 3)) < 0.03] = 0.0
    rays["dir"] = d
    rays["tmax"] = rng.choice([0.0, 8.0, 256.0, 700.0], n)
    rays["kind"] = rng.choice([0, 1, 2, 3, 256, 257, 258, 259], n)
    p = vg.default_params(7, frame=2.0)
    t = q.default_tuning()
    t.sort, t.refill_min = sort, 32
    _, out, shadow = q.run(dw, rays, p, tuning=t)
    t.sort, t.refill_min = 0, 8                       # lane by lane, unsorted
    _, lanes, lane_shadow = q.run(dw, rays, p, tuning=t)
    want = vg.trace(dw, rays, p)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert torch.equal(lanes, want)
    assert torch.equal(shadow, lane_shadow)
    assert int((vg.shadows(shadow)["traced"] == 1).sum()) > 0
