"""FP64 MinSR solve at the edges of the blocked factorisation: orders around the 32-wide blocks,
one block, and orders with more tiles than CTAs; both solve spaces, against the oracle's update."""
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


def step(nqs, N, M, Ns, space, seed):
    from spin_based_neural_network_gb300 import abi
    cfg = abi.config_defaults(ansatz=abi.ANSATZ_RBM, rbm_hidden_units=M, hamiltonian=abi.HAM_TFIM, sr_diag_shift=1e-2,
                              learning_rate=0.01)
    rng = np.random.default_rng(seed)
    a = nqs.Ansatz(cfg, N)
    p0 = rng.normal(0.0, 0.2, size=a.P)
    a.params[:] = p0
    batch = np.where(rng.random((Ns, N)) < 0.5, 1, -1).astype(np.int32)
    nqs.set_options(fp64_space=space)
    try:
        info, E, d = nqs.sr_step_batch(cfg, N, 1, a, batch, minsr=True, log_amp_fn=a.log_amp_fn, user=a.user)
    finally:
        nqs.set_options()
    amp = O.Amp(O.OR_RBM, N, M, p0)
    E0, d0, _ = O.minsr_step(O.ham(O.OR_TFIM, N, 1), amp, batch, 1e-2, 0.01)
    assert info.converged == 1
    return float(np.linalg.norm(d - d0) / max(np.linalg.norm(d0), 1e-300))    # one sample: both are zero


# the parity bar of the FP64 update: 1e-10 relative
@pytest.mark.parametrize("Ns", [1, 2, 8, 31, 32, 33, 63, 64, 65, 255, 256, 257, 700])
def test_sample_space_orders(nqs, Ns):
    from spin_based_neural_network_gb300 import abi
    assert step(nqs, 10, 7, Ns, abi.SPACE_SAMPLES, Ns) < 1e-10


@pytest.mark.parametrize("N,M,Ns", [(3, 2, 40), (5, 5, 200), (8, 7, 300), (12, 20, 600)])
def test_parameter_space_orders(nqs, N, M, Ns):
    from spin_based_neural_network_gb300 import abi
    assert step(nqs, N, M, Ns, abi.SPACE_PARAMETERS, M) < 1e-10


def test_order_with_more_tiles_than_ctas(nqs):
    from spin_based_neural_network_gb300 import abi
    assert step(nqs, 12, 8, 1633, abi.SPACE_SAMPLES, 5) < 1e-10


def test_barrier_timeout_returns_an_error(nqs):
    from spin_based_neural_network_gb300 import abi
    assert nqs.lib().nqs_gpu_set_barrier_budget(1) == 0
    try:
        with pytest.raises(nqs.NqsError):
            step(nqs, 10, 7, 700, abi.SPACE_SAMPLES, 1)
        assert "grid barrier timed out" in nqs.last_error()
    finally:
        assert nqs.lib().nqs_gpu_set_barrier_budget(0) == 0
    assert step(nqs, 10, 7, 700, abi.SPACE_SAMPLES, 1) < 1e-10
