"""Trainer.loss over an epoch: one tensor from construction on, with the last
batch's block losses in it, also where the batch size is lowered afterwards
(fewer blocks than the buffer has room for)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BATCH = 256


@pytest.fixture(scope="module")
def env(geometry):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from orgpu import learned, pipeline
    rng = np.random.default_rng(8)
    x = torch.from_numpy(rng.normal(0, 1.5, 3 * BATCH * 16).astype(np.float32)).cuda()
    y = torch.from_numpy((rng.random(3 * BATCH) < 0.2).astype(np.uint8)).cuda()
    rc = pipeline.Reconstruction(geometry[0], 0, max_events=1)
    return learned.Learned(rc), x, y


def _trainer(env, n):
    from orgpu import learned
    lr, x, y = env
    sp = learned.ScorerParams.init(np.zeros(16, np.float32), np.ones(16, np.float32), seed=2)
    return learned.Trainer(lr, sp, x[:n * 16], y[:n], batch=BATCH, pos_weight=3.0)


def test_loss_keeps_its_tensor(env):
    t = _trainer(env, BATCH)
    held = t.loss
    assert held.shape == (t.nblk,) and float(held.abs().sum()) == 0.0
    for _ in range(2):
        loss = t.epoch(np.random.default_rng(1))
        assert t.loss is held
        # one batch: its block losses are the epoch's
        assert loss > 0 and float(held.sum()) == loss


def test_loss_is_the_last_batch(env):
    """Over three batches: what the last one alone gives from the parameters
    that the first two leave."""
    import torch
    from orgpu import _lib
    t, u = _trainer(env, 3 * BATCH), _trainer(env, 3 * BATCH)
    held = t.loss
    t.epoch(np.random.default_rng(5))
    perm = np.random.default_rng(5).permutation(3 * BATCH)
    last = None
    for b in range(3):
        idx = torch.from_numpy(perm[b * BATCH:(b + 1) * BATCH]).cuda()
        last = torch.zeros(u.nblk, device="cuda")
        _lib.check(u.lib.or_mlp_gradient(u.ctx, u.model.ptr(), u.features.data_ptr(), u.labels.data_ptr(),
                                         idx.data_ptr(), BATCH, u.pos_weight, u.grad.data_ptr(), last.data_ptr(),
                                         u.stream), "or_mlp_gradient")
        _lib.check(u.lib.or_mlp_adam(u.ctx, u.param.data_ptr(), u.m1.data_ptr(), u.m2.data_ptr(), u.grad.data_ptr(),
                                     u.nblk, b + 1, u.lr, 0.9, 0.999, 1e-8, u.model.ptr(), u.stream), "or_mlp_adam")
        torch.cuda.synchronize()
    assert np.array_equal(held.cpu().numpy(), last.cpu().numpy())


def test_smaller_batch_afterwards(env):
    """128 rows a batch: one block, the rest of the buffer adds nothing."""
    import torch
    t, u = _trainer(env, BATCH), _trainer(env, BATCH)
    t.batch = u.batch = BATCH // 2
    torch.full((4, 2), float("nan"), device="cuda")  # freed memory that is not zero
    a, b = t.epoch(np.random.default_rng(3)), u.epoch(np.random.default_rng(3))
    assert a == b and 0.0 < a < 10.0
