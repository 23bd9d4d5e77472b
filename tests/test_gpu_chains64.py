"""FP64 Philox chains of the RBM / complex RBM against the oracle's chains, sample for sample: hidden
widths around the warp's lane counts, both move sets, ragged batches, sharply peaked states, and
weights beyond the product form's range (run through log|psi|)."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nqs():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import nqs as N
    N.set_options()
    return N


def chains(nqs, kind, Lx, Ly, M, scale, exchange, C, n, decor, seed):
    from spin_based_neural_network_gb300 import abi
    N = Lx * Ly
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=M, rng_seed=seed, num_thermalize=37, num_decorrelate=decor)
    a = nqs.Ansatz(cfg, N)
    a.params[:] = np.random.default_rng(seed).normal(0.0, scale, size=a.P)
    n_down = N // 2 if exchange else -1
    s = nqs.Sampler(N, cfg, a.log_amp_fn, a.user,
                    nqs.options(num_chains=C, rng=abi.RNG_PHILOX, move=int(exchange), n_down=n_down, lattice_x=Lx,
                                lattice_y=Ly, square_pbc=1))
    s.thermalize()
    got = s.batch(n)
    amp = O.Amp(kind, N, M, a.params.copy())
    want, _, acc, pro = O.chain_sampler(amp, O.ham(O.OR_HEIS, Lx, Ly, pbc=1), seed, C, int(exchange), n_down, 37,
                                        -(-n // C), decor)
    assert np.array_equal(got, want[:n])
    if n % C == 0:
        assert s.acceptance_ratio() == pytest.approx(acc / pro, abs=0)


@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 16, 17, 32, 33, 65, 129, 192, 256])
@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
def test_widths(nqs, kind, M):
    for exchange in (False, True):
        chains(nqs, kind, 5, 2, M, 0.2, exchange, 5, 17, 3, 100 + M)


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("scale", [0.7, 3.0, 40.0])
def test_peaked_states_and_weights_out_of_range(nqs, kind, scale):
    for exchange in (False, True):
        chains(nqs, kind, 4, 4, 24, scale, exchange, 7, 35, 11, 5)


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("M", [1, 5, 16])
@pytest.mark.parametrize("scale", [0.02, 0.8, 2.5, 60.0])
def test_two_proposals_a_round(nqs, kind, M, scale):
    # nearly free chains (both proposals accepted), peaked ones, and weights out of range; an odd
    # number of moves, records at every move and across the 32-move draws
    chains(nqs, kind, 9, 1, M, scale, False, 6, 6 * 41, 1, 11)
    chains(nqs, kind, 4, 4, M, scale, False, 3, 3 * 5, 31, 12)
