"""Local energies of a single site, whose lattice has no bonds: 0, with and without a symmetry projection."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("ham", [1, 2, 4])
@pytest.mark.parametrize("projected", [False, True])
def test_single_site(kind, ham, projected):
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import abi, nqs
    nqs.set_options()
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=3, hamiltonian=ham, j2_coupling=0.5, j_z_coupling=1.3)
    a = nqs.Ansatz(cfg, 1)
    fn, user = a.log_amp_fn, a.user
    if projected:
        sym = nqs.Symproj(fn, user, 1, np.zeros((1, 1), np.int32), np.ones(1))
        fn, user = sym.log_amp_fn, sym.user
    e = nqs.local_energy_batch(cfg, 1, 1, np.array([[1], [-1]], np.int32), fn, user)
    assert np.array_equal(e, np.zeros(2))
