"""The training kernel at the edges of its tiling (128 rows a tile, one CTA per
SM): a single row, a tile less, full and more, one row beyond a whole wave of
tiles, rows that do not start on 16 bytes, and a drawn minibatch smaller than
its tile.  Checked against the numpy restatement with the same BF16-rounded
operands; what is left is FP32 accumulation order (bounds of the row sums:
relative 2^-24 times the square root of the rows, far below 5e-4)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, seed, shift=0):
    import torch

    g = torch.Generator().manual_seed(seed)
    x = torch.randn(n, 96, generator=g) * 0.5
    x[:, 82:] = 0.0
    y = torch.randint(0, 154, (n,), generator=g).to(torch.uint8)
    flat = torch.empty(n * 96 + shift, dtype=torch.bfloat16, device="cuda")
    xd = flat[shift:].view(n, 96)
    xd.copy_(x)
    return xd, y.cuda()


@pytest.mark.parametrize("n,shift", [(1, 0), (127, 0), (128, 1), (129, 0), (152 * 128 + 1, 0)])
def test_gradients_at_tile_edges(lib, n, shift):
    import mlp_oracle as mo
    from ecmgenerator_gb300 import proposal as P

    m = P.ProposalModel(seed=3)
    x, y = _data(n, 5 + n, shift)
    loss, g = m.loss_grad(x, y)
    want_loss, want = mo.loss_grad(m.get_params(), x.float().cpu().numpy(), y.cpu().numpy(), bf16_operands=True)
    assert abs(loss - want_loss) < 1e-5 * max(1.0, abs(want_loss))
    got, ref = P.split_params(g), P.split_params(np.asarray(want))
    for k in got:
        assert np.linalg.norm(got[k] - ref[k]) <= 5e-4 * np.linalg.norm(ref[k]), k
    m.close()


def test_training_steps_repeat_and_do_not_depend_on_logging(lib):
    from ecmgenerator_gb300 import proposal as P

    x, y = _data(900, 2)
    out = []
    for log in (True, True, False):
        m = P.ProposalModel(seed=3)
        loss, acc = m.train(x, y, steps=5, batch=300, lr=1e-3, seed=8, log=log)
        out.append(m.get_params())
        if log:
            assert np.all(np.isfinite(loss)) and np.all((acc >= 0) & (acc <= 1))
        m.close()
    # the gradient sums have a fixed order: the same bits every time
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
