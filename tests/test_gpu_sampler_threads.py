"""FP64 Philox samplers of several host threads, each with a sampler and an ansatz of its own of another size, draw
what they draw alone."""
import threading

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def test_threads():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import abi, nqs
    nqs.set_options()

    def sampler(k):
        N, M = (8, 12, 20, 30)[k], (5, 40, 70, 130)[k]
        cfg = abi.config_defaults(ansatz=O.OR_CRBM if k % 2 else O.OR_RBM, rbm_hidden_units=M, rbm_init_scale=0.3,
                                  rng_seed=k + 1, num_thermalize=10, num_decorrelate=3)
        a = nqs.Ansatz(cfg, N)
        return a, nqs.Sampler(N, cfg, a.log_amp_fn, a.user, nqs.options(num_chains=64, rng=abi.RNG_PHILOX))

    def draw(s, out):
        for _ in range(40):
            out.append(s.batch(256))

    alone, together = [[] for _ in range(4)], [[] for _ in range(4)]
    made = [sampler(k) for k in range(4)]
    for k in range(4):
        draw(made[k][1], alone[k])
    made = [sampler(k) for k in range(4)]
    threads = [threading.Thread(target=draw, args=(made[k][1], together[k])) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x, y in zip(alone, together):
        assert len(y) == 40 and all(np.array_equal(p, q) for p, q in zip(x, y))


def test_beside_mixed_steps():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import abi, nqs
    cfg = abi.config_defaults(ansatz=O.OR_CRBM, rbm_hidden_units=16, rbm_init_scale=0.1, rng_seed=5, num_decorrelate=3,
                              num_thermalize=10, hamiltonian=abi.HAM_HEISENBERG, sr_diag_shift=1e-3, learning_rate=0.0)
    spins = np.where(np.random.default_rng(5).random((512, 16)) < 0.5, 1, -1).astype(np.int32)
    a, b = nqs.Ansatz(cfg, 16), nqs.Ansatz(cfg, 16)
    nqs.set_options(precision=abi.PREC_MIXED)
    try:
        def step():
            return nqs.sr_step_batch(cfg, 4, 4, a, spins)[1]

        def sampler():
            return nqs.Sampler(16, cfg, b.log_amp_fn, b.user, nqs.options(num_chains=64, rng=abi.RNG_PHILOX))

        E, s, t = [step(), step()], sampler(), sampler()      # the steps' graph is captured before the threads run
        alone, together = [s.batch(256) for _ in range(60)], [t.batch(256)]
        thread = threading.Thread(target=lambda: together.extend(t.batch(256) for _ in range(59)))
        thread.start()
        while thread.is_alive():
            E.append(step())
        thread.join()
    finally:
        nqs.set_options()
    assert all(np.array_equal(x, y) for x, y in zip(alone, together)) and len(together) == 60
    assert all(np.array_equal(x, E[0]) for x in E)
