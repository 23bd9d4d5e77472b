"""A mixed step that fails behind the fork of its energy statistics (its 200000 x 200000 system does not fit) leaves
the following step on the same buffers as it would be without it."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def test_step_after_a_failed_mixed_step():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import abi, nqs
    cfg = abi.config_defaults(ansatz=O.OR_CRBM, rbm_hidden_units=2, rbm_init_scale=0.3, hamiltonian=abi.HAM_HEISENBERG,
                              sr_diag_shift=1e-3, learning_rate=0.01, sr_cg_max_iters=200, sr_cg_tol=1e-12)
    spins = np.where(np.random.default_rng(5).random((200000, 8)) < 0.5, 1, -1).astype(np.int32)
    a = nqs.Ansatz(cfg, 8)
    start = a.params.copy()

    def step(batch, **options):
        a.params[:] = start
        nqs.set_options(**options)
        try:
            info, E, _ = nqs.sr_step_batch(cfg, 8, 1, a, batch, minsr=bool(options))
        finally:
            nqs.set_options()
        return np.array(E), a.params.copy()

    E0, p0 = step(spins[:1000])
    for _ in range(4):
        with pytest.raises(nqs.NqsError):
            step(spins, precision=abi.PREC_MIXED)
        E, p = step(spins[:1000])
        assert np.array_equal(E, E0) and np.array_equal(p, p0)
