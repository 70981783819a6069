"""Walks that pass the lower iteration cap: long ones, and ones that return to
a state they were in (ended at once with the full cap's step count), for
every kind of ray and iteration caps around the lower cap and the stretches
after it, bit-exact against the oracle, which takes every iteration."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

DIMS = (64, 16, 512)


@pytest.fixture(scope="module")
def long_rays():
    """Rays of 150 and more steps, those that reach the cap first."""
    import voxelg_b200 as vg
    ow = po.World(*DIMS)
    terrain = vg.TerrainParams(seed=5, base_height=24.0, amplitude=20.0, water_level=16)
    ow.generate(terrain)
    rng = np.random.default_rng(1)
    n = 2_000_000
    r = np.zeros(n, po.RAY)
    # far from the window corner and along z, where landings round coarsest
    r["org"] = rng.uniform([0, 20, 1500], [256, 64, 2048], (n, 3))
    d = rng.normal(size=(n, 3))
    d[:, 0] *= 10.0 ** rng.uniform(-4, 0, n)
    d[:, 1] *= 10.0 ** rng.uniform(-4, 0, n)
    r["dir"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["tmax"] = 700.0
    r["kind"] = rng.integers(0, 3, n)
    p = vg.default_params(7)
    steps = po.trace_batch(ow, r, p)[0].view(po.RECORD)["steps"]
    capped = steps == np.where(r["kind"] == 1, p.any_max_iters, p.max_iters)
    assert capped.sum() >= 3
    keep = np.concatenate([np.flatnonzero(capped), np.flatnonzero(~capped & (steps > 150))[:4000]])
    return ow, terrain, r[keep]


@pytest.mark.parametrize("cap", [1, 179, 180, 181, 239, 240, 241, 300, 768, 1024, 5000])
def test_every_cap(long_rays, cap):
    import torch
    import voxelg_b200 as vg
    from voxelg_b200 import queue
    ow, terrain, rays = long_rays
    dw = vg.DeviceWorld(*DIMS)
    dw.generate(terrain)
    for flags in (1, 7):
        p = vg.default_params(flags)
        p.max_iters = p.any_max_iters = cap
        want = po.trace_batch(ow, rays, p)[0].view(po.RECORD)
        got = vg.records(vg.trace(dw, rays, p))
        assert got.tobytes() == want.tobytes(), (cap, flags)
        for refill in (32, 8):
            t = queue.default_tuning()
            t.refill_min = refill
            _, out, _ = queue.run(dw, rays, p, t, with_shadow=False)
            torch.cuda.synchronize()
            assert vg.records(out).tobytes() == want.tobytes(), (cap, flags, refill)
    dw.close()
