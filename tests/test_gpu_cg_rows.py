"""CG-SR with the Jacobian's rows in shared memory, at the edges of its splits: rows per CTA and
parameters per thread at their boundaries, one sample, the holomorphic pair of matrices, and shapes
just past what fits (the kernel that streams the Jacobian).  Capped at 10 iterations, against the
oracle's update."""
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


def step(nqs, kind, N, M, Ns, holo, iters=10):
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
    return float(np.linalg.norm(d - d0) / max(np.linalg.norm(d0), 1e-300))


# the parity bar of the FP64 update: 1e-10 relative
@pytest.mark.parametrize("N,M,Ns", [(4, 3, 1), (4, 3, 5), (6, 5, 64), (15, 15, 300), (16, 15, 608), (16, 15, 609),
                                    (10, 46, 257), (20, 24, 1030), (20, 48, 700), (30, 65, 200), (30, 66, 200)])
def test_shapes(nqs, N, M, Ns):
    assert step(nqs, O.OR_RBM, N, M, Ns, False, 3 if Ns < 10 else 10) < 1e-10


@pytest.mark.parametrize("N,M,Ns", [(6, 5, 64), (12, 19, 333), (12, 39, 1024), (12, 64, 1500)])
def test_holomorphic(nqs, N, M, Ns):
    assert step(nqs, O.OR_CRBM, N, M, Ns, True) < 1e-10
