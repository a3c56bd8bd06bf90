"""Training targets in any contiguous shape whose first rows are the batch's moves."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("shape", [lambda y: y.reshape(-1), lambda y: y.reshape(-1, 2, 16),
                                   lambda y: torch.cat([y, y.flip(0)])])
def test_target_shapes(shape):
    from adock_b200.proposal import IN, ProposalNet
    net = ProposalNet(DEV, seed=1)
    g = torch.Generator(device=DEV).manual_seed(2)
    x = torch.randn(70, IN, device=DEV, generator=g).to(torch.bfloat16)
    y = torch.randn(70, 32, device=DEV, generator=g)
    y[:, 26] = 7
    y[:, 27:] = 0
    grads = net.loss_grad(x, y)[1]
    assert all(torch.equal(a, b) for a, b in zip(grads, net.loss_grad(x, shape(y))[1]))
