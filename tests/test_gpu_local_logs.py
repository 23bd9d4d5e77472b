"""FP64 local energies of moves beyond the products' range (through log 2 cosh of the units) over the widths of a
lane, flips and pair flips, against the definition in extended precision."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_local_prod import energies

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nqs():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import nqs as N
    N.set_options()
    return N


# |log psi| of a few 10^3 as at M = 40 and 8.0: exp(log ratio) carries 8 x 2^-53 x 4e3 = 4e-12 relative
@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("M", [31, 33, 65, 130, 256])
def test_widths(nqs, kind, M):
    for ham in (0, 2):
        e, r = energies(nqs, kind, M, ham, 4, 3, 320.0 / M, 25, M)
        assert np.all(np.isfinite(r.real))
        assert np.max(np.abs(e - r) / np.maximum(np.abs(r), 1.0)) < 1e-11
