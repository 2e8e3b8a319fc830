"""Adam steps on drawn minibatches against a host restatement: the rows
(splitmix64 of the step's seed and the row, modulo n), the mean loss and the
hits, and the weights.  FP64 with the matrix-product operands rounded to BF16,
as tests of the gradient have it.

Bounds.  The gradient is good to 5e-4 of its norm there.  Adam's first step is
the learning rate times the gradient's sign; of entries that are spread like a
normal distribution, that error reaches past zero for 2e-4, whose step is then
off by twice its length: 2 sqrt(2e-4) = 3e-2 of the change of all weights, 6e-2
allowed over three steps.  Where such an entry goes changes the loss in second
order only (1e-4).  A row drawn wrongly, a parameter that takes another's
gradient or a wrong bias correction is off by a third or more.  A logit's
rounding may decide one hit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(seed, batch, n):
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, batch + 1, dtype=np.uint64)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return (z % np.uint64(n)).astype(np.int64)


@pytest.mark.parametrize("n,batch", [(1, 1), (1, 300), (7, 100), (1024, 128), (4099, 1), (4099, 300), (1 << 17, 129),
                                     (1000003, 640)])
def test_steps_equal_the_restatement(lib, n, batch):
    import mlp_oracle as mo
    import torch
    from ecmgenerator_gb300.proposal import ProposalModel

    steps, lr, seed = 3, 1e-3, 0xFFFFFFFFFFFF0000 + n  # wraps
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    x = torch.randn((n, 96), generator=g, device="cuda") * 0.5
    x[:, 82:] = 0.0
    x = x.to(torch.bfloat16)
    y = torch.randint(0, 160, (n,), generator=g, device="cuda").to(torch.uint8)
    m = ProposalModel(seed=5)
    w0 = m.get_params().astype(np.float64)
    loss, acc = m.train(x, y, steps=steps, batch=batch, lr=lr, seed=seed)
    got = m.get_params().astype(np.float64)
    m.close()

    w, m1, m2 = w0.copy(), np.zeros_like(w0), np.zeros_like(w0)
    for t in range(1, steps + 1):
        r = torch.from_numpy(_rows((seed + 0x51ED27 * t) % 2**64, batch, n)).cuda()
        xb, yb = x[r].float().cpu().numpy(), y[r].cpu().numpy()
        want, grad = mo.loss_grad(w, xb, yb, bf16_operands=True)
        assert abs(loss[t - 1] - want) <= (1e-5 if t == 1 else 1e-4) * max(1.0, want), t
        b = mo._bf16
        W1, b1, W2, b2, W3, b3 = mo.split(w)
        a = mo.gelu(b(xb) @ b(W1) + b1)
        z = b(mo.gelu(b(a) @ b(W2) + b2)) @ b(W3) + b3
        hits = np.sum(z.argmax(1) == yb)
        assert abs(acc[t - 1] * batch - hits) <= np.bincount(r.cpu().numpy()).max() + 0.5  # one row's draws
        m1 = 0.9 * m1 + 0.1 * grad
        m2 = 0.999 * m2 + 0.001 * grad * grad
        w = w - lr * (m1 / (1.0 - 0.9**t)) / (np.sqrt(m2 / (1.0 - 0.999**t)) + 1e-8)
    assert np.linalg.norm(got - w) <= 6e-2 * np.linalg.norm(w - w0)
