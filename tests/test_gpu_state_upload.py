"""A state uploaded right after bafqmc_create is the state the chains hold: the handle's memory is
cleared in the order of its own stream, so the clearing cannot overtake the upload."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_state_uploaded_at_once_survives_the_clearing_of_a_large_handle():
    from bafqmc_b200 import solver
    from bafqmc_b200.calibrate_tau import workload_6x6_beta8

    p, chains = workload_6x6_beta8(), 2048
    rng = np.random.default_rng(3)
    seeds = (2 * rng.integers(1, 2 ** 30 - 1, chains) + 1).astype(np.int32)
    phi = rng.standard_normal(chains * p.Ltrot * p.Lq * 2)
    got_seeds, got = np.empty_like(seeds), np.empty_like(phi)
    for _ in range(4):
        with solver.Ensemble([p], np.zeros(chains, dtype=np.int32)) as ens:
            ens.set_state_flat(seeds, phi)
            ens.get_state_flat(got_seeds, got)
        assert np.array_equal(got_seeds, seeds) and np.array_equal(got, phi)
