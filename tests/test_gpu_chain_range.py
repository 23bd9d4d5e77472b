"""FP64 Philox chains at the edges of the product form's range, against the oracle's chains, sample for
sample: weights whose factors overflow a double while the theta and the moves' sums stay small, and
parameters that are not finite."""
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


def compare(nqs, kind, Lx, Ly, M, fill, exchange, C=6, n_spc=9, decor=7):
    from spin_based_neural_network_gb300 import abi
    N = Lx * Ly
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=M, rng_seed=23, num_thermalize=13, num_decorrelate=decor)
    a = nqs.Ansatz(cfg, N)
    a.params[:] = np.random.default_rng(3).normal(0.0, 0.05, size=a.P)
    fill(a.params)
    n_down = N // 2 if exchange else -1
    s = nqs.Sampler(N, cfg, a.log_amp_fn, a.user,
                    nqs.options(num_chains=C, rng=abi.RNG_PHILOX, move=int(exchange), n_down=n_down, lattice_x=Lx,
                                lattice_y=Ly, square_pbc=1))
    s.thermalize()
    got = s.batch(n_spc * C)
    amp = O.Amp(kind, N, M, a.params.copy())
    want, _, acc, pro = O.chain_sampler(amp, O.ham(O.OR_HEIS, Lx, Ly, pbc=1), 23, C, int(exchange), n_down, 13, n_spc, decor)
    assert np.array_equal(got, want)
    assert s.acceptance_ratio() == pytest.approx(acc / pro, abs=0)


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("M", [2, 3, 20, 40])
@pytest.mark.parametrize("w", [60.0, 89.0, 140.0, 176.0, 220.0])
def test_opposite_units(nqs, kind, M, w):
    # two hidden units whose weights on sites 0 and 1 are opposite: the signed sums of every move vanish
    # while exp(4 (W_u - W_v)) of one unit passes exp(709) from w = 89 (exchanges) or 178 (flips)
    def fill(p):
        W = p[4 + M:4 + M + 4 * M].reshape(M, 4)
        W[:2] = [[w, -w, 0.0, 0.0], [-w, w, 0.0, 0.0]]
        W[2:, :] *= 0.2
    for exchange in (False, True):
        compare(nqs, kind, 4, 1, M, fill, exchange)


@pytest.mark.parametrize("M", [5, 20])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("part,imag", [("bias", False), ("bias", True), ("weight", False), ("weight", True), ("visible", True)])
def test_parameters_that_are_not_finite(nqs, M, bad, part, imag):
    N = 8
    k = {"visible": 3, "bias": N + 2, "weight": N + M + 2 * N + 3}[part] + (N + M + M * N if imag else 0)

    def fill(p):
        p[k] = bad
    for exchange in (False, True):
        compare(nqs, O.OR_CRBM, 4, 2, M, fill, exchange)
