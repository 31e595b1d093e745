"""bafqmc_net_set_tensor_cores on lattices where only the weight gradients run on the tensor cores (width 64, but
no tiling of the convolutions): off and on again is the state the network was created in.  A batch this small has
one block to a weight's sum, so the weights' gradients have no order of additions and are compared bit for bit; a
bias is added up by four groups of threads, in any order, and stays out of that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lx,ly,L", [(3, 3, 20), (5, 1, 32), (2, 2, 24)])
def test_off_and_on_again(lx, ly, L):
    from bafqmc_b200.proposer import Proposer, init_params, layer_shapes
    params = init_params(64, 4)
    rng = np.random.default_rng(5)
    tail = 27 * 4 * 64 + 4
    params[-tail:-4] = rng.uniform(-0.05, 0.05, tail - 4).astype(np.float32)
    phi, target = rng.standard_normal((2, 2, L, lx * ly, 2))
    weights = np.concatenate([np.r_[np.ones(27 * ci * co, bool), np.zeros(co, bool)] for ci, co in layer_shapes(64)])
    with Proposer(lx, ly, L, params=params) as net:
        g = [net.loss_grad(phi, target)[1]]
        for enable in (False, True):
            net.set_tensor_cores(enable)
            g.append(net.loss_grad(phi, target)[1])
    assert not np.array_equal(g[0][weights], g[1][weights])   # other kernels
    np.testing.assert_array_equal(g[0][weights], g[2][weights])
    assert np.linalg.norm(g[1] - g[0]) <= 1e-5 * np.linalg.norm(g[0])
