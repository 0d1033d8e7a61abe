"""A training step whose pipeline gave up: NaN gradients and loss, nothing
updated, and the next step as if it had not been.  The failure is made on the
host, by the mark that a block whose waits ran out leaves in the work area."""
import numpy as np
import pytest

from .test_gpu_learned import _params

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FAILED = 0x4D4C502067617665             # FFA_MLP_STEP_FAILED


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")


def mark(tr):
    a = (-tr.work.data_ptr() % 128) // 4
    tr.work[a:a + 2].view(torch.int64).fill_(FAILED)


@pytest.mark.parametrize("mode", ["host", "schedule", "graph"])
@pytest.mark.parametrize("B", [64, 1000])
def test_failed_step_updates_nothing(B, mode):
    from pyffa_b200 import learned
    rng = np.random.default_rng(B)
    x, t = np.zeros((B, 8), np.float32), np.zeros((B, 8), np.float32)
    x[:, :6] = rng.uniform(-1, 1, (B, 6))
    t[:, :6] = x[:, :6] + 0.05 * rng.standard_normal((B, 6))
    x, t = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    lr = None if mode == "host" else torch.tensor([1e-3, 2e-3, 3e-3, 4e-3])
    trainers = []
    for _ in range(2):
        p = torch.from_numpy(learned.from_dict(_params(7))).cuda()
        trainers.append(learned.Trainer(p, batch=B, freeze_skip=False, lr_table=lr))
    a, b = trainers

    def step(tr):
        if mode == "graph":
            tr.graph_step(x, t)
        else:
            tr.step(x, t, 1e-3)
    for tr in trainers:
        step(tr)
        step(tr)                         # "graph": a replay
    state = [v.clone() for v in (a.p, a.m, a.v)] + ([a.counter.clone()] if lr is not None else [])
    mark(a)
    step(a)
    if mode == "host":
        a.t -= 1                         # the host's count of Adam steps
    torch.cuda.synchronize()
    assert bool(torch.isnan(a.g).all()) and bool(torch.isnan(a.loss_part).all())
    for v, w in zip(state, (a.p, a.m, a.v, a.counter)):
        assert torch.equal(v, w)
    step(a)
    step(b)
    for v, w in zip((a.p, a.g, a.m, a.v, a.loss_part), (b.p, b.g, b.m, b.v, b.loss_part)):
        assert torch.equal(v, w)
    if lr is not None:
        assert int(a.counter) == int(b.counter) == 3


@pytest.mark.parametrize("fail", [False, True])
def test_training_run_reports_it(fail, monkeypatch):
    from pyffa_b200 import learned
    rng = np.random.default_rng(1)
    X = np.zeros((4096, 8), np.float32)
    X[:, :5] = rng.uniform(-1, 1, (4096, 5))
    X = torch.from_numpy(X).cuda()
    T = X + 0.05 * torch.sin(3 * X)
    plain, calls = learned.Trainer.graph_step, []

    def graph_step(tr, x, t):
        calls.append(1)
        if fail and len(calls) == 3:
            mark(tr)
        plain(tr, x, t)
    monkeypatch.setattr(learned.Trainer, "graph_step", graph_step)
    p = torch.from_numpy(learned.init_params(0)).cuda()
    if fail:
        with pytest.raises(RuntimeError, match="1 of 8 training steps gave up"):
            learned.train(p, X, T, epochs=2, batch=1024)
    else:
        learned.train(p, X, T, epochs=2, batch=1024)
    assert bool(torch.isfinite(p).all())
