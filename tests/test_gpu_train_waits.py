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
