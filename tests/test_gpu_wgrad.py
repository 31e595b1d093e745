"""The tensor-core weight gradient (width 64) at its edges: fewer slices than a staged run of 32, a remainder of
it, exactly one, lattices that are their own neighbours, and more pairs than one block takes; against the oracle.

Tolerance: activations and their gradients are rounded to bf16 (half an ulp is 2^-9) at six places between the
input and a weight's gradient on both sides, and sums in another order flip some of those roundings: 6 x 2^-9 =
1.2e-2 if every one of a small batch's goes the same way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lx,ly,L,batch", [(1, 1, 3, 2), (1, 2, 16, 1), (2, 2, 17, 3), (3, 2, 32, 2), (2, 3, 33, 2),
                                           (4, 4, 64, 9), (1, 3, 700, 2)])
def test_gradient_against_oracle(lx, ly, L, batch):
    from bafqmc_b200.proposer import Proposer, init_params
    from oracle import proposer as P
    rng = np.random.default_rng(5)
    params = init_params(64, 4)
    tail = 27 * 4 * 64 + 4
    params[-tail:-4] = rng.uniform(-0.05, 0.05, tail - 4).astype(np.float32)
    phi = rng.standard_normal((batch, L, lx * ly, 2)).astype(np.float32).astype(np.float64)
    target = rng.standard_normal(phi.shape).astype(np.float32).astype(np.float64)
    with Proposer(lx, ly, L, width=64, params=params) as net:
        _, grad = net.loss_grad(phi, target)
    _, ref = P.loss_and_grad(params, phi, target, lx, ly, rounding=True)
    off = 0
    for ci, co in P.layer_shapes(64):
        for n in (27 * co * ci, co):   # the weights, then the biases
            d, r = grad[off:off + n] - ref[off:off + n], ref[off:off + n]
            assert np.linalg.norm(d) <= 1.2e-2 * np.linalg.norm(r), (ci, co, n)
            off += n
