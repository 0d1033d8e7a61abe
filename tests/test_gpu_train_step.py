"""The fused training step at the edges of its tiles.

Gradients of every parameter and the loss against the oracle for batches
around the 64-sample tile, one that leaves the least room in the work area
and one with more tiles than SMs, every output count, a sixth input, and
inputs that are only 4-byte aligned; nothing may be written past the work area.
Tolerances: those of the batch-512 test (bfloat16 operands and the hardware
tanh), which do not depend on the batch."""
import numpy as np
import pytest

from oracle import mlp as M

from .test_gpu_learned import _params, _rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")


def unaligned(a):
    """The array on the device, 4 bytes past an aligned address."""
    buf = torch.empty(a.size + 1, dtype=torch.float32, device="cuda")
    v = buf[1:].view(a.shape)
    v.copy_(torch.from_numpy(a))
    return v


@pytest.mark.parametrize("B,n_fit", [(1, 4), (63, 1), (64, 4), (65, 6), (129, 4), (961, 5), (1024, 4), (19_001, 4)])
def test_gradients_and_loss(B, n_fit):
    from pyffa_b200 import learned
    d = _params(30 + n_fit)
    rng = np.random.default_rng(B)
    x, t = np.zeros((B, 8), np.float32), np.zeros((B, 8), np.float32)
    x[:, :6] = rng.uniform(-1, 1, (B, 6))
    t[:, :6] = x[:, :6] + 0.05 * rng.standard_normal((B, 6))
    tr = learned.Trainer(torch.from_numpy(learned.from_dict(d)).cuda(), batch=B, n_fit=n_fit, freeze_skip=False)
    size = tr.work.numel()
    room = torch.full((size + 4096,), 7.0, dtype=torch.float32, device="cuda")
    tr.work = room[:size]
    tr.step(unaligned(x), unaligned(t), 0.0)
    torch.cuda.synchronize()
    assert bool((room[size:] == 7.0).all())
    g = learned.to_dict(tr.g.cpu().numpy())
    x6, t6 = x[:, :6].astype(np.float64), t[:, :6].astype(np.float64)
    sse16, g16 = M.loss_and_grads(d, x6, t6, n_fit=n_fit, bf16_ops=True)
    _, g64 = M.loss_and_grads(d, x6, t6, n_fit=n_fit)
    assert abs(tr.loss_part.sum().item() - sse16) <= 3e-3 * sse16
    for k in g16:
        assert _rel(g[k], g16[k]) <= 1e-2, (k, _rel(g[k], g16[k]))
        assert _rel(g[k], g64[k]) <= 5e-2, (k, _rel(g[k], g64[k]))
    full = tr.g.cpu().numpy()
    used = learned.from_dict(g)
    assert np.array_equal(full, used)              # padded entries are zero
