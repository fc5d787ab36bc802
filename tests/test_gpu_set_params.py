"""Weights set from pageable memory are the ones that the next pass uses: a
network given another's weights has its gradients bit for bit, every time."""
import pytest

from poker_trainer_b200.mlp import LeafNet

pytestmark = pytest.mark.gpu


def test_weights_are_there_before_their_copies_are_made(gpu):
    import torch
    g = torch.Generator().manual_seed(3)
    x, t = torch.randn(33, 300, generator=g).cuda(), torch.randn(33, 130, generator=g).cuda()
    nets = [LeafNet(300, 256, 3, 130, max_batch=33, seed=s) for s in (1, 2)]
    params, want = [n.params() for n in nets], []
    for n in nets:
        n.backward(x, t)
        want.append(n.grad_tensor().clone())
    for k in range(20):
        nets[0].set_params(params[k % 2].copy())
        nets[0].backward(x, t)
        assert torch.equal(nets[0].grad_tensor(), want[k % 2])
