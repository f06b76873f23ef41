"""The network's fused passes at the sizes where their tiling can go wrong:
row tiles of 128 (one row, a tile and one row, more tiles than the device holds
pairs of blocks, an odd number of them), columns split between two blocks
unevenly or not at all, outputs up to the limit, weight-gradient parts that
start inside a row tile -- and one network too wide for them, which runs layer
by layer.  Against an FP32 restatement with the weights, inputs and hidden
activations rounded to BF16 where the kernels store them in BF16.

Tolerances, from BF16's unit roundoff u = 2^-9: an output is a sum over
`width` products of rounded values whose own rounding the restatement repeats;
what differs is the FP32 summation order (2^-24 per term) and the BF16 flips
it causes in the activations of each layer, at most u of a value each, averaging
over the width: 2 u of the largest output is far above it and far below any
misplaced tile, column or row.  Gradients round dZ to BF16 once a layer, in the
kernels alone: u per element and layer, 3e-2 of the norm bounds 7 layers of it."""
import numpy as np
import pytest
import torch

from oneflow_b200.mlp import MLP

pytestmark = pytest.mark.gpu


def bf16(t):
    return t.to(torch.bfloat16).to(torch.float32)


def restate(net, flat, x):
    h = bf16(x)
    layers = []
    o = 0
    for k, n in net.layer_shapes():
        layers.append((flat[o:o + k * n].view(k, n), flat[o + k * n:o + k * n + n]))
        o += k * n + n
    for i, (w, b) in enumerate(layers):
        z = h @ (w + (bf16(w) - w).detach()) + b
        h = torch.nn.functional.gelu(z) if i + 1 < len(layers) else z
        if i + 1 < len(layers):
            h = h + (bf16(h) - h).detach()
    return h


def rows_of(n, k, seed):
    g = torch.Generator().manual_seed(seed)
    return (torch.rand((n, k), generator=g) * 2 - 1).cuda()


@pytest.mark.parametrize("shape,rows", [((8, 16, 1, 1), 1), ((8, 48, 3, 4), 129), ((22, 256, 6, 4), 128),
                                        ((22, 256, 6, 4), 128 * 150 + 5), ((256, 208, 2, 100), 500),
                                        ((17, 64, 4, 128), 333), ((8, 272, 2, 4), 200), ((8, 64, 2, 130), 200)])
def test_predictions(shape, rows):
    net = MLP(*shape, seed=3)
    p = net.params()
    p = p + np.random.default_rng(1).uniform(-0.05, 0.05, p.shape).astype(np.float32)   # biases too
    net.set_params(p)
    x = rows_of(rows, shape[0], 2)
    y = net.predict(x)
    ref = restate(net, torch.tensor(p, device="cuda"), x)
    assert (y - ref).abs().max().item() < 2 * 2.0 ** -9 * ref.abs().max().item()


@pytest.mark.parametrize("shape,rows", [((8, 16, 1, 1), 64), ((8, 48, 3, 17), 1344), ((22, 256, 6, 4), 192),
                                        ((22, 256, 6, 4), 8192), ((100, 208, 2, 100), 4160), ((8, 272, 2, 4), 192)])
def test_loss_and_gradient(shape, rows):
    net = MLP(*shape, seed=5)
    x, y = rows_of(rows, shape[0], 3), rows_of(rows, shape[3], 4)
    loss, g = net.loss_grad(x, y)
    flat = torch.tensor(net.params(), device="cuda", requires_grad=True)
    ref = ((restate(net, flat, x) - y) ** 2).mean()
    ref.backward()
    assert abs(loss - ref.item()) < 1e-3 * ref.item()
    r = flat.grad.cpu().numpy()
    assert np.linalg.norm(g - r) < 3e-2 * np.linalg.norm(r)


def test_training_step_is_adam_on_the_gradient_and_the_next_pass_uses_it():
    # one step on a batch drawn from a single sample: every row the same, so
    # the gradient is that of loss_grad on it; Adam's first step moves each
    # weight by lr g / (|g| + eps sqrt(c2)), and the loss of the second step is
    # the new weights' (both packings refreshed)
    net, lr = MLP(22, 256, 3, 4, seed=7), 1e-3
    x, y = rows_of(1, 22, 5), rows_of(1, 4, 6)
    p0 = net.params()
    _, g = net.loss_grad(x.repeat(64, 1).contiguous(), y.repeat(64, 1).contiguous())
    losses = net.train(x, y, 1, batch=64, lr=lr, seed=1)
    p1 = net.params()
    big = np.abs(g) > 1e-6
    assert np.abs((p1 - p0)[big] + lr * np.sign(g[big])).max() < 0.02 * lr   # eps / |g| <= 1e-2
    after, _ = net.loss_grad(x.repeat(64, 1).contiguous(), y.repeat(64, 1).contiguous())
    again = net.train(x, y, 1, batch=64, lr=lr, seed=1)
    assert losses[0] > after and abs(again[0] - after) < 1e-6 * after
