"""The gradient kernel at the edges of its 32-node blocks, 16-node warps and
1024-node chunks, against the CPU restatement."""
import numpy as np
import pytest

from icflow_b200.warm_start import MLP, NI, NO, init_params
from oracle.mlp_oracle import loss_and_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 1023, 1025, 8193, 20011])
def test_gradient_at_block_edges(n):
    rng = np.random.default_rng(n)
    p = init_params(1)
    p[-195:] = rng.normal(0, 0.2, 195).astype(np.float32)
    norm = np.concatenate([rng.normal(0, 0.2, NI), 0.5 + rng.random(NI), np.ones(NO)]).astype(np.float32)
    x = rng.normal(size=(n, NI)).astype(np.float32)
    t = rng.normal(size=(n, NO)).astype(np.float32)
    net = MLP()
    net.set_params(p, norm)
    g, loss = net.grad(x, t)
    lref, gref = loss_and_grad(p, norm, x, t)
    net.close()
    # float32 sums over the nodes in 32-node, then 1024-node, then chunk order:
    # at most 32 + 32 + n / 1024 roundings of 2^-24 of the sum of magnitudes,
    # which the signs of the terms let exceed the sum by about sqrt(n); the
    # test of the whole gradient allows 1e-5 of its largest entry
    assert abs(loss - lref) <= 1e-5 * lref
    assert np.abs(g - gref).max() <= 1e-5 * np.abs(gref).max()
