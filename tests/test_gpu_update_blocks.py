"""Edges of the blocked local update and of the FP64 tensor-pipe products: lattices whose site count leaves
a short last block (of 8 slots), a single block, a remainder of the 8 x 8 tiles or of the four-k steps, in
every size class and both sectors, against the oracle.

Tolerance: the tests that compare the same quantities elsewhere take 1e-10 of the largest entry of G; a
sweep here is at most 20 slices with stabilisation every 5, so rounding of a different order of additions
(n slots of 1e-16 per element and slice) stays below 1e-12; 1e-11 is asserted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NC = [(1, 2), (3, 3), (2, 4), (2, 5), (4, 4), (1, 17), (5, 5), (4, 7), (3, 11), (5, 7), (6, 6), (1, 37), (5, 8), (7, 9),
      (8, 8), (8, 9), (1, 73)]
PAIR = [(2, 2), (1, 4), (1, 5), (2, 3), (2, 4), (3, 3), (2, 6), (1, 17), (3, 6), (1, 19), (5, 5), (5, 7), (6, 6)]


def _compare(op, sp, seeds):
    from bafqmc_b200 import solver
    from oracle import oracle as O
    with solver.Ensemble([sp], [0] * len(seeds)) as ens:
        ens.fields_from_seeds(seeds)
        ens.pre()
        ens.sweep(1)
        got_seeds, got_phi = ens.get_state()
        _, _, chains = O.init_chains(op, seeds=seeds)
        for c, ch in enumerate(chains):
            ch.pre()
            ch.sweep_bin()
            G = ens.green(c)
            ref = ch.prop.Gr
            if sp.sector == 1:
                G = solver.nambu_green(G)
            assert int(got_seeds[c]) == ch.seed
            assert np.array_equal(got_phi[c], ch.phi)
            assert np.max(np.abs(G - ref)) <= 1e-11 * np.max(np.abs(ref))


def _kw(lx, ly, L, nwrap, shift):
    return dict(U1=1.0, U2=-0.5, mu=-7.0, Nlx=lx, Nly=ly, Ltrot=L, Beta=0.05 * L, NlxTherm=lx, NlyTherm=ly, LtrotTherm=L,
                Nwrap=nwrap, Nbin=1, Nsweep=1, shiftLoc=shift, iniType=2, iniAmpl=1.0)


@pytest.mark.parametrize("lx,ly", NC)
def test_number_conserving_sizes(lx, ly):
    from bafqmc_b200.params import SolverParams
    from oracle import oracle as O
    kw = _kw(lx, ly, 10, 5, 1.5)
    _compare(O.Params(**kw), SolverParams(**kw), [11, 12])


@pytest.mark.parametrize("lx,ly", PAIR)
def test_nambu_sizes(lx, ly):
    from bafqmc_b200.params import SolverParams
    from oracle import oracle as O
    kw = _kw(lx, ly, 10, 5, 1.0)
    _compare(O.Params(**kw, RDelta=0.25, pairing=True), SolverParams(**kw, delta=0.25, sector=1), [21, 22])


@pytest.mark.parametrize("U1,U2", [(1.0, 0.0), (0.0, -0.5)])
def test_one_channel(U1, U2):
    """Only one HS channel active: the fields staged for both serve the one."""
    from bafqmc_b200.params import SolverParams
    from oracle import oracle as O
    kw = dict(_kw(5, 3, 10, 5, 1.5), U1=U1, U2=U2)
    _compare(O.Params(**kw), SolverParams(**kw), [31])
