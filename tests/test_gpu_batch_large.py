"""A batch instance past the order from which the preconditioner is applied by blocked substitution (4608), whose
trailing tiles have no tensor maps as the single system's do: the same step as the single system."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ns", [4608, 4801])
def test_matches_the_single_step(Ns):
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import abi, nqs
    cfg = abi.config_defaults(ansatz=abi.ANSATZ_RBM, rbm_hidden_units=144, rbm_init_scale=0.2, hamiltonian=abi.HAM_TFIM,
                              rng_seed=7, num_samples=Ns, num_thermalize=64, num_decorrelate=36, sr_diag_shift=1e-2,
                              learning_rate=0.02, transverse_field=1.1)
    o = nqs.options(num_chains=1024, rng=abi.RNG_PHILOX, lattice_x=6, lattice_y=6, square_pbc=1,
                    precision=abi.PREC_MIXED, fp32_estimator=1)

    def instance():
        a = nqs.Ansatz(cfg, 36)
        s = nqs.Sampler(36, cfg, a.log_amp_fn, a.user, o)
        s.thermalize()
        return a, s

    nqs.set_options(square_pbc=1, precision=abi.PREC_MIXED, fp32_estimator=1, refine_sweeps=20)
    try:
        (a, s), (b, t) = instance(), instance()
        start = a.params.copy()
        B = nqs.Batch([(cfg, 6, 6, a, s, None, None)])
        info = B.step()[0]
        one = nqs.sr_step_minsr(cfg, 6, 6, b, t, b.log_amp_fn, b.user)
        B.free()
    finally:
        nqs.set_options()
    assert info.converged == 1 and one.converged == 1
    assert info.mean_energy == pytest.approx(one.mean_energy, rel=1e-12)
    # both solves stop at a residual of 1e-10; a condition of 1e5 at most at this shift
    assert np.max(np.abs(a.params - b.params)) <= 1e-5 * np.max(np.abs(b.params - start))
