"""The self-energy network's block kernels (hidden width 128) at the edges of
their tiles: 128-row blocks, 128-wide input and output blocks, a batch of one
row, output layers of more than two blocks.  The checker rounds the same
operands to BF16 and sums in FP64; activations that round differently move a
result by one BF16 step (2^-8) of a few of their terms, so 1e-2 of the largest.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import mlp_ref  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out,batch", [(1, 1, 1), (128, 128, 128), (127, 129, 127), (129, 127, 257),
                                              (385, 513, 640)])
def test_blocks_match_checker(pkg, n_in, n_out, batch):
    rng = np.random.default_rng(n_in + batch)
    net = pkg.surrogate.MLP(n_in, n_out, hidden=128, seed=2)
    dims = [n_in, 128, 128, 128, n_out]
    p = net.params()
    off = 0
    for i in range(4):
        off += dims[i] * dims[i + 1]
        p[off:off + dims[i + 1]] = rng.normal(scale=0.1, size=dims[i + 1])
        off += dims[i + 1]
    net.set_params(p)
    x = rng.normal(size=(batch, n_in)).astype(np.float32)
    t = rng.normal(size=(batch, n_out)).astype(np.float32)
    y_ref = mlp_ref.forward(p, dims, x)[0]
    assert np.abs(net.forward(x).cpu().numpy() - y_ref).max() < 1e-2 * np.abs(y_ref).max()
    g, loss = net.gradients(x, t)
    g_ref, loss_ref = mlp_ref.gradients(p, dims, x, t)
    assert abs(loss - loss_ref) < 1e-2 * loss_ref
    off = 0
    for i in range(4):
        for n in (dims[i] * dims[i + 1], dims[i + 1]):
            assert np.linalg.norm(g[off:off + n] - g_ref[off:off + n]) < 2e-2 * np.linalg.norm(g_ref[off:off + n]), i
            off += n
    # the gradients leave the weights alone; a training step moves each by the
    # learning rate at most (first Adam step) and repeats on the same start
    assert np.array_equal(net.params(), p)
    import torch

    xd, td = torch.as_tensor(x, device="cuda"), torch.as_tensor(t, device="cuda")
    net.train_step(xd, td, 1e-3)
    p1 = net.params()
    assert 0 < np.abs(p1 - p).max() <= 1.001e-3
    net.set_params(p)
    net.train_step(xd, td, 1e-3)
    assert np.array_equal(net.params(), p1)
