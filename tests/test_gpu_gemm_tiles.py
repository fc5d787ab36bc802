"""Every tile of the GEMM's dispatch (gemm_shape, mlp.cu) at one and many steps
of its ring, with each epilogue, against fp32 products of the same bf16
operands; and the training step's reductions and transposes at batch sizes
that leave padded rows, against the fp32 gradients with the kernels' rounding
points (tolerances as tests/test_gpu_mlp.py's: f32 accumulation of bf16
products 1e-5 of the largest, a bf16 result 1e-2)."""
import numpy as np
import pytest

from poker_trainer_b200.mlp import LeafNet, gemm_bf16
from test_gpu_mlp import reference_gradients

pytestmark = pytest.mark.gpu

# (m, n): tiles 32, 64, 128 alone on an SM, and 128 two to an SM.
SHAPES = [(128, 256), (768, 1024), (1024, 1536), (1664, 1536)]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("k", [64, 704])
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
def test_tiles(gpu, m, n, k, epi):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n + k + epi)
    a = (torch.randn(m, k, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    b = (torch.randn(n, k, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda", generator=g)
    zin = torch.randn(m, n, device="cuda", generator=g).to(torch.bfloat16)
    acc = a.double() @ b.double().T
    c, z = gemm_bf16(a, b, epi, bias if epi in (1, 2) else None, zin if epi == 3 else None)
    pre = acc + bias.double()
    x = zin.double()
    ref = {0: acc, 1: pre, 2: torch.nn.functional.gelu(pre),
           3: acc * (0.5 * (1 + torch.erf(x / np.sqrt(2))) + x * torch.exp(-0.5 * x * x) / np.sqrt(2 * np.pi))}[epi]
    tol = 1e-5 if epi < 2 else 1e-2
    assert float((c.double() - ref).abs().max()) <= tol * float(ref.abs().max())
    if epi == 2:
        assert float((z.double() - pre).abs().max()) <= 1e-2 * float(pre.abs().max())


# Steps of 64, 128 and 192 of K: a last step that is partly empty, and rings that
# go round; 256 x 2688: tiles 32 wide, two to an SM.
@pytest.mark.parametrize("m,n", SHAPES + [(256, 2688)])
@pytest.mark.parametrize("k", [256, 1344])
@pytest.mark.parametrize("epi", [0, 2])
def test_steps(gpu, m, n, k, epi):
    test_tiles(gpu, m, n, k, epi)


@pytest.mark.parametrize("rows", [1, 129, 300])
@pytest.mark.parametrize("masked", [False, True])
def test_gradients_with_padded_rows(gpu, rows, masked):
    import torch
    net = LeafNet(70, 128, 2, 200, max_batch=rows, seed=3)
    g = torch.Generator().manual_seed(rows)
    x, t = torch.randn(rows, 70, generator=g), torch.randn(rows, 200, generator=g)
    mask = (torch.rand(rows, 200, generator=g) > 0.4).float() if masked else torch.ones(rows, 200)
    ref = reference_gradients(net, net.params(), x, t, mask)
    loss = net.backward(x.cuda(), t.cuda(), mask.cuda() if masked else None)
    got = net.grad_tensor().cpu().numpy()
    assert abs(loss - ref[0]) <= 2e-2 * abs(ref[0])
    for (w, b), (rw, rb) in zip(net.split(got), ref[1]):
        for u, v in ((w, rw), (b, rb)):
            v = np.asarray(v, np.float32)
            assert np.linalg.norm(u - v) <= 2e-2 * max(np.linalg.norm(v), 1e-12)
    # One Adam step moves every real weight, and the network's next pass uses it.
    y0 = net.forward(x.cuda())
    net.adam_step(1e-2)
    assert not torch.equal(y0, net.forward(x.cuda()))
