"""The training kernel's bounded waits made to run out by a small poll limit, at
whatever wait that limit reaches (the forward chains with one poll, later ones
with more): a call either reports ECMG_ERR_BOUND or gives the bits of a call
without a limit, and the call after it is an ordinary one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITS = [1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 128, 512]


def _rows(n, seed=4):
    import torch

    g = torch.Generator().manual_seed(seed)
    x = torch.randn(n, 96, generator=g) * 0.5
    x[:, 82:] = 0.0
    return x.to(torch.bfloat16).cuda(), torch.randint(0, 154, (n,), generator=g).to(torch.uint8).cuda()


def test_gradient_with_short_waits(lib):
    import torch

    from ecmgenerator_gb300._lib import EcmgError
    from ecmgenerator_gb300.proposal import ProposalModel

    m = ProposalModel(seed=3)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x, y = _rows(2 * sms * 128 + 1)  # a second and a third tile per CTA: weight gradients in flight
    loss, grad = m.loss_grad(x, y)
    ran_out = 0
    for limit in LIMITS:
        assert lib.ecmg_mlp_set_wait_limit(m.h, limit) == 0
        try:
            got = m.loss_grad(x, y)
        except EcmgError as e:
            assert e.status == 3  # ECMG_ERR_BOUND
            ran_out += 1
            assert lib.ecmg_mlp_set_wait_limit(m.h, 0) == 0
            got = m.loss_grad(x, y)
        assert got[0] == loss and np.array_equal(got[1], grad), limit
    assert ran_out > 0
    m.close()


def test_training_takes_whole_steps_only(lib):
    """a step whose gradient is not whole changes neither the weights nor Adam's
    state or step count, and neither do the steps queued behind it: what is left
    to do, done afterwards, ends in the bits of an undisturbed run"""
    import ctypes

    from ecmgenerator_gb300.proposal import ProposalModel

    steps, batch, lr, seed = 6, 700, 1e-3, 8
    x, y = _rows(5000)
    m = ProposalModel(seed=3)
    start = m.get_params()
    want_loss, want_acc = m.train(x, y, steps=steps, batch=batch, lr=lr, seed=seed)
    want = m.get_params()
    m.close()
    for limit in LIMITS:
        m = ProposalModel(seed=3)
        assert lib.ecmg_mlp_set_wait_limit(m.h, limit) == 0
        loss, acc = np.zeros(steps, np.float32), np.zeros(steps, np.float32)
        rc = lib.ecmg_mlp_train(m.h, x.data_ptr(), y.data_ptr(), 5000, steps, batch, lr, ctypes.c_ulonglong(seed),
                                loss.ctypes.data, acc.ctypes.data)
        done = int(np.sum(~np.isnan(loss)))
        assert rc == (0 if done == steps else 3), limit
        assert np.array_equal(loss[:done], want_loss[:done]) and np.array_equal(acc[:done], want_acc[:done])
        assert np.isnan(loss[done:]).all() and np.isnan(acc[done:]).all()
        if limit == 1:
            assert done == 0
        if done == 0:
            assert np.array_equal(m.get_params(), start)
        assert lib.ecmg_mlp_set_wait_limit(m.h, 0) == 0
        m.train(x, y, steps=steps - done, batch=batch, lr=lr, seed=seed)
        assert np.array_equal(m.get_params(), want), limit
        m.close()
