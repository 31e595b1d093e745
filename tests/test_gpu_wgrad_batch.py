"""A batch of 65536 (chain, site) pairs, more than a grid's second dimension holds, for the tensor-core weight
gradient: a batch that repeats a few configurations has their gradient.

Tolerance: repetition by a power of two scales every activation gradient exactly, and on a single site a block
takes one configuration in either batch, so that only the float32 additions of the blocks' sums differ.  There
are 65536 of them in an element of the large batch, each off by half a unit (2^-24) of a partial sum that is at
most the sum of the magnitudes: 2^16 x 2^-24 = 2^-8 of the configurations' mean magnitude, and the smaller
batch's four additions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_gradient_of_a_repeated_batch():
    from bafqmc_b200.proposer import Proposer, init_params
    L, base, rep = 321, 4, 16384
    params = init_params(64, 4)
    rng = np.random.default_rng(7)
    tail = 27 * 4 * 64 + 4
    params[-tail:-4] = rng.uniform(-0.05, 0.05, tail - 4).astype(np.float32)
    phi = rng.standard_normal((base, L, 1, 2))
    target = rng.standard_normal(phi.shape)
    with Proposer(1, 1, L, width=64, params=params) as net:
        loss0, grad0 = net.loss_grad(phi, target)
        single = sum(np.abs(net.loss_grad(phi[b:b + 1], target[b:b + 1])[1].astype(np.float64)) for b in range(base)) / base
        loss, grad = net.loss_grad(np.tile(phi, (rep, 1, 1, 1)), np.tile(target, (rep, 1, 1, 1)))
    assert abs(loss - loss0) <= 1e-9 * abs(loss0)
    assert single.max() > 0
    d = np.abs(grad.astype(np.float64) - grad0)
    assert np.all(d <= (2.0 ** -8 + 2.0 ** -21) * single), (d - 2.0 ** -8 * single).max()
