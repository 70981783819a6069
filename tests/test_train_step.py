"""The training step where its tiles of 32 samples go round the device more than
once: both groups of every CTA, several tiles a group, a ragged last tile, a
batch that is not 16-byte aligned."""
import numpy as np
import pytest

from oracle import mlp as om

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prop():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    import voxelg_b200 as vg
    from voxelg_b200 import learned as vl
    dw = vg.DeviceWorld(64, 16, 64)
    p = vl.Proposal(dw, seed=3)
    yield p
    p.close()
    dw.close()


# On 148 SMs: one tile more than there are CTAs, one more than there are groups,
# the default batch, the same with a ragged end, three and a half tiles a group.
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("batch", [4737, 9473, 16384, 16389, 32768 + 31])
def test_gradient(prop, batch, offset):
    """Against the oracle's float64 step.  The longest chain of additions behind
    a gradient entry is about 80 + 64 + 64 + 112 + 148 + 8 < 500 roundings of
    2^-24 relative to what has been added up, 3e-5; three times that of the
    tensor's largest entry is allowed.  Twice the same batch: the same bits."""
    import torch
    rng = np.random.default_rng(batch)
    X = rng.uniform(-1, 1, (batch, om.N_IN)).astype(np.float32)
    X[:, 70:] = 0
    X[:, 6:70] = rng.integers(0, 2, (batch, 64))
    y = rng.uniform(1, 6.5, batch).astype(np.float32)
    room = torch.zeros(batch * om.N_IN + 1, dtype=torch.float32, device="cuda")
    x = room[offset:offset + batch * om.N_IN].view(batch, om.N_IN)
    x.copy_(torch.from_numpy(X))
    t = torch.from_numpy(y).cuda()
    torch.cuda.synchronize()
    loss, g = prop.grad(x, t)
    loss2, g2 = prop.grad(x, t)
    assert loss == loss2 and np.array_equal(g.view(np.uint32), g2.view(np.uint32))
    rl, rg = om.loss_and_grad(prop.params().astype(np.float64), X, y)
    assert abs(loss - rl) <= 1e-5 * abs(rl)
    o = 0
    for name, shape in om.SIZES:
        n = int(np.prod(shape))
        a, b = g[o:o + n], rg[o:o + n]
        assert np.max(np.abs(a - b)) <= 1e-4 * np.max(np.abs(b)), name
        o += n
