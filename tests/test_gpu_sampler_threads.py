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
