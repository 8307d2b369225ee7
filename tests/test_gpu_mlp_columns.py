"""The surrogate's column inputs and the step's loss against the paths they replaced.

loglik(theta, rt, choice) reads its three arrays where they are; the values and the
gradients are those of the joined rows, bit for bit, at sizes around the tiles' edges
and for strided, double and integer inputs.  A training step's loss is the mean of
the per-block losses (a sum of at most 148 float32 values in another order: each of
its additions may round by 2^-24 of the total, 148 * 2^-24 < 1e-5).
"""

import numpy as np
import pytest
import torch

from ssms_b200.surrogate import MlpSurrogate, SurrogateLogLik

pytestmark = pytest.mark.gpu


def _rows(n, seed=3):
    g = np.random.default_rng(seed)
    x = np.concatenate([g.uniform(-1, 1, (n, 5)), g.uniform(0.1, 3, (n, 1)), g.choice([-1.0, 1.0], (n, 1))], axis=1)
    return torch.from_numpy(x.astype(np.float32)).cuda()


@pytest.mark.parametrize("n", [0, 1, 127, 128, 129, 148 * 128 + 1, 2 * 148 * 128 + 5, 5 * 148 * 128 - 1])
def test_columns_agree_with_joined_rows(cuda, n):
    net, x = MlpSurrogate("angle", seed=1), _rows(n)
    rows = x.clone().requires_grad_(True)
    want = SurrogateLogLik.apply(rows, net)
    w = torch.linspace(-1, 2, n, device="cuda")
    (gx,) = torch.autograd.grad((want * w).sum(), rows)
    th, rt, ch = (t.clone().requires_grad_(True) for t in (x[:, :5], x[:, 5], x[:, 6]))
    got = net.loglik(th, rt, ch)
    gt, gr, gc = torch.autograd.grad((got * w).sum(), (th, rt, ch))
    assert torch.equal(got, want) and torch.equal(gt, gx[:, :5]) and torch.equal(gr, gx[:, 5]) and torch.equal(gc, gx[:, 6])
    with torch.no_grad():  # views with strides, and another type
        assert torch.equal(net.loglik(x[:, :5], x[:, 5:6], x[:, 6].double()), want)
        assert torch.equal(net.forward(x), want)
    net.check()


def test_unequal_row_counts_are_refused(cuda):
    net, x = MlpSurrogate("angle", seed=1), _rows(4)
    with pytest.raises(RuntimeError):
        net.loglik(x[:, :5], x[:3, 5], x[:, 6])


@pytest.mark.parametrize("n", [1, 127, 8192, 148 * 128 + 77])
def test_step_loss_is_the_mean_of_the_block_losses(cuda, n):
    net = MlpSurrogate("angle", seed=2)
    rec = torch.cat([_rows(n), torch.randn(n, 1, device="cuda")], dim=1)
    _, lpart, k = net.grad(rec)
    want = float(lpart[:k].double().sum()) / n
    loss = net.train_step(rec)
    assert loss.shape == () and loss.dtype == torch.float32
    np.testing.assert_allclose(float(loss), want, rtol=1e-5)
