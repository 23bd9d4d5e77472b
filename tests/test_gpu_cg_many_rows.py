"""CG-SR of many samples of few parameters: a CTA's row dots (R samples, 2 R of the holomorphic pair)
just within, just past and several times its 256 threads.  At most 10 iterations (5 where there are only
19 or 38 parameters), against the oracle's update."""
import ctypes as C

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


def step(nqs, kind, N, M, Ns, holo, iters):
    from spin_based_neural_network_gb300 import abi
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=M, hamiltonian=abi.HAM_TFIM, sr_diag_shift=1e-2,
                              learning_rate=0.01, sr_cg_max_iters=iters, sr_cg_tol=1e-30)
    rng = np.random.default_rng(Ns + M)
    a = nqs.Ansatz(cfg, N)
    p0 = rng.normal(0.0, 0.1, size=a.P)
    a.params[:] = p0
    batch = np.where(rng.random((Ns, N)) < 0.5, 1, -1).astype(np.int32)
    info, E, d = nqs.sr_step_batch(cfg, N, 1, a, batch, minsr=2 if holo else 0, log_amp_fn=a.log_amp_fn, user=a.user)
    amp = O.Amp(kind, N, M, p0)
    f = O.holo_step if holo else O.cgsr_step
    E0, d0, i0 = f(O.ham(O.OR_TFIM, N, 1), amp, batch, 1e-2, 0.01, iters, 1e-30)
    assert info.cg_iterations == i0.cg_iterations
    return float(np.linalg.norm(d - d0) / np.linalg.norm(d0))


# the parity bar of the FP64 update: 1e-10 relative
@pytest.mark.parametrize("kind,N,M,rows,iters", [(O.OR_RBM, 8, 8, 256, 10), (O.OR_RBM, 8, 8, 257, 10), (O.OR_RBM, 8, 8, 264, 10),
                                                 (O.OR_RBM, 4, 3, 600, 5), (O.OR_CRBM, 8, 4, 128, 10), (O.OR_CRBM, 8, 4, 129, 10),
                                                 (O.OR_CRBM, 4, 3, 300, 5)])
def test_rows_per_cta(nqs, kind, N, M, rows, iters):
    sms = C.c_int()
    assert nqs.lib().nqs_gpu_device_info(None, 0, C.byref(sms)) == 0
    assert step(nqs, kind, N, M, rows * sms.value, kind == O.OR_CRBM, iters) < 1e-10
