"""loglik without gradients runs the forward kernel alone.

Inputs that ask for gradients do not get them under no_grad: no row of
derivatives may be computed or kept.  The forward pass allocates its output
(4 bytes a row; the derivatives would be 28 more), so the peak of the call's
allocations tells the two apart.
"""

import pytest
import torch

from ssms_b200.surrogate import MlpSurrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_no_derivatives_without_gradients(cuda, mode):
    n = 1 << 18
    net = MlpSurrogate("angle", seed=1)
    theta = torch.rand(n, 5, device="cuda", requires_grad=True)
    rt, choice = torch.rand(n, device="cuda"), torch.ones(n, device="cuda")
    want = net.loglik(theta, rt, choice)
    assert want.requires_grad
    with mode():
        net.loglik(theta, rt, choice)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        got = net.loglik(theta, rt, choice)
        peak = torch.cuda.max_memory_allocated() - before
    assert not got.requires_grad
    assert torch.equal(got, want.detach())
    assert peak < 8 * n
    (g,) = torch.autograd.grad(want.sum(), theta)
    assert g.shape == theta.shape
