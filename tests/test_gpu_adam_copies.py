"""The bf16 copies of the weights that an Adam step writes (one per layout, 64 x
64 weights a block, up to 8 layers a launch) against the copies that set_params
makes of the same f32 weights: a network given the other's weights has the same
gradients bit for bit, which read both copies."""
import numpy as np
import pytest

from poker_trainer_b200.mlp import LeafNet

pytestmark = pytest.mark.gpu


# One hidden layer; layers of 128 and 384 columns; ten layers (two launches).
@pytest.mark.parametrize("inputs,hidden,layers,outputs", [(70, 128, 1, 200), (300, 256, 3, 130), (60, 128, 9, 40)])
def test_copies_after_adam(gpu, inputs, hidden, layers, outputs):
    import torch
    g = torch.Generator().manual_seed(layers)
    x, t = torch.randn(33, inputs, generator=g).cuda(), torch.randn(33, outputs, generator=g).cuda()
    a = LeafNet(inputs, hidden, layers, outputs, max_batch=33, seed=1)
    b = LeafNet(inputs, hidden, layers, outputs, max_batch=33, seed=2)
    before = a.params()
    for _ in range(2):
        a.backward(x, t)
        a.adam_step(1e-2)
    after = a.params()
    for (w0, b0), (w1, b1) in zip(a.split(before), a.split(after)):
        w0, w1 = np.asarray(w0), np.asarray(w1)  # padded: zeros, which stay
        assert np.all(w1[w0 == 0] == 0) and np.mean(w0[w0 != 0] != w1[w0 != 0]) > 0.9
        assert np.any(np.asarray(b0) != np.asarray(b1))
    b.set_params(after)
    a.backward(x, t)
    b.backward(x, t)
    assert torch.equal(a.grad_tensor(), b.grad_tensor())
