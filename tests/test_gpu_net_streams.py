"""A network's own stream and a handle's stream do not wait for each other by themselves: a first learned move
on buffers that are still being cleared, network calls right after a move or a collection whose kernels are
still queued, against the same calls with everything finished in between.  Equal bits, as the kernels are the
same; the loss is a double that many blocks add to, so it may differ by their order (1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHAINS = 1024


@pytest.fixture(scope="module")
def setup():
    from bafqmc_b200 import solver
    from bafqmc_b200.params import SolverParams
    from bafqmc_b200.proposer import init_params
    p = SolverParams(U1=1.0, U2=-0.5, mu=-6.0, Nlx=6, Nly=6, Ltrot=32, Beta=1.6, NlxTherm=6, NlyTherm=6, LtrotTherm=32,
                     Nwrap=8, Nbin=1, Nsweep=1, shiftLoc=1.5, iniType=2, iniAmpl=1.0)
    rng = np.random.default_rng(17)
    params = init_params(64, 2)
    tail = 27 * 4 * 64 + 4
    params[-tail:-4] = rng.uniform(-0.01, 0.01, tail - 4).astype(np.float32)
    seeds = (2 * rng.integers(1, 2 ** 30 - 1, CHAINS) + 1).astype(np.int32)
    phi = rng.standard_normal(CHAINS * 32 * 36 * 2)
    with solver.Ensemble([p], np.zeros(CHAINS, dtype=np.int32)) as ens:
        yield ens, params, seeds, phi


def _start(ens, seeds, phi):
    ens.set_state_flat(seeds, phi)
    ens.pre()
    ens.synchronize()


def _net(params):
    from bafqmc_b200.proposer import Proposer
    return Proposer(6, 6, 32, params=params)


def _state(ens):
    s, f = np.empty(CHAINS, np.int32), np.empty(CHAINS * 32 * 36 * 2)
    ens.get_state_flat(s, f)
    return s, f


def test_first_move_of_a_new_network(setup):
    ens, params, seeds, phi = setup
    got = []
    for ready in (True, False):
        _start(ens, seeds, phi)
        with _net(params) as net:
            if ready:
                net.forward(np.zeros((CHAINS, 32, 36, 2)))
            acc, hst = ens.learned_move(net)
        got.append((acc, hst, *_state(ens)))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_network_call_behind_a_queued_move(setup):
    ens, params, seeds, phi = setup
    x = np.random.default_rng(3).standard_normal((CHAINS, 32, 36, 2))
    got = []
    for wait in (True, False):
        _start(ens, seeds, phi)
        with _net(params) as net:
            ens.learned_move(net, want=False)
            if wait:
                ens.synchronize()
            out = net.forward(x)
        got.append((out, *_state(ens)))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_training_behind_a_queued_collection(setup):
    ens, params, seeds, phi = setup
    losses = []
    for wait in (True, False):
        _start(ens, seeds, phi)
        with _net(params) as net:
            net.reserve(CHAINS, 2)
            for _ in range(2):
                ens.sweep(1)
                net.collect(ens)
            if wait:
                ens.synchronize()
            losses.append(net.train(1, 64, 1, 1e-3, seed=5)[0])
    assert abs(losses[1] - losses[0]) <= 1e-12 * abs(losses[0])


def test_move_captured_on_the_handles_stream(setup):
    """A handle's stream under capture takes no wait on the network's own stream, which is outside the capture."""
    import ctypes as C
    ens, params, seeds, phi = setup
    cu = C.CDLL("libcuda.so.1")
    stream = C.c_void_p(ens.stream)
    got = []
    with _net(params) as net:
        _start(ens, seeds, phi)
        ens.learned_move(net)   # allocates
        for capture in (False, True):
            _start(ens, seeds, phi)
            net.status()
            if capture:
                graph, run = C.c_void_p(), C.c_void_p()
                assert cu.cuStreamBeginCapture_v2(stream, 2) == 0   # relaxed
                ens.learned_move(net, want=False)
                assert cu.cuStreamEndCapture(stream, C.byref(graph)) == 0
                assert cu.cuGraphInstantiateWithFlags(C.byref(run), graph, C.c_ulonglong(0)) == 0
                assert cu.cuGraphLaunch(run, stream) == 0
            else:
                ens.learned_move(net, want=False)
            ens.synchronize()
            got.append(_state(ens))
            if capture:
                assert cu.cuGraphExecDestroy(run) == 0 and cu.cuGraphDestroy(graph) == 0
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
