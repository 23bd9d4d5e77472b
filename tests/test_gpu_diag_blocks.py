"""Mixed solve at orders that leave partial 16-column panels and partial 64-wide diagonal blocks: the
update against the FP64 parameter-space solve of the same batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nqs():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import nqs as N
    N.set_options()
    return N


# the bar of the mixed solve with the FP64 estimator: 1e-8 relative
@pytest.mark.parametrize("Ns", [2, 15, 16, 17, 33, 47, 63, 64, 65, 79, 127, 129, 177, 191, 400])
def test_orders(nqs, Ns):
    from spin_based_neural_network_gb300 import abi
    N, M = 16, 12
    cfg = abi.config_defaults(ansatz=abi.ANSATZ_RBM, rbm_hidden_units=M, hamiltonian=abi.HAM_TFIM, sr_diag_shift=1e-2,
                              learning_rate=0.01)
    rng = np.random.default_rng(Ns)
    a = nqs.Ansatz(cfg, N)
    p0 = rng.normal(0.0, 0.3, size=a.P)
    batch = np.where(rng.random((Ns, N)) < 0.5, 1, -1).astype(np.int32)
    d = {}
    try:
        for name, kw in (("mixed", dict(precision=abi.PREC_MIXED, mixed_space=abi.SPACE_SAMPLES, refine_sweeps=20)),
                         ("fp64", dict(precision=abi.PREC_FP64, fp64_space=abi.SPACE_PARAMETERS))):
            nqs.set_options(**kw)
            a.params[:] = p0
            info, E, d[name] = nqs.sr_step_batch(cfg, N, 1, a, batch, minsr=True, log_amp_fn=a.log_amp_fn, user=a.user)
            assert info.converged == 1
            if name == "mixed":
                assert nqs.last_step_stats().mixed_fallback == 0
    finally:
        nqs.set_options()
    assert np.linalg.norm(d["mixed"] - d["fp64"]) < 1e-8 * np.linalg.norm(d["fp64"])
