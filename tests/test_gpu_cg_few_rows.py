"""CG-SR of few samples of many parameters: CTAs that hold no rows share the columns.  Fewer iterations than the rank of
the centred rows, against the oracle's update."""
import pytest

import oracle_lib as O
from test_gpu_cg_many_rows import step

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nqs():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import nqs as N
    N.set_options()
    return N


# the parity bar of the FP64 update: 1e-10 relative
@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("N,M", [(8, 4), (16, 15), (16, 55), (15, 62)])
@pytest.mark.parametrize("Ns,iters", [(2, 1), (4, 2), (5, 3), (17, 5), (65, 5)])
def test_few_samples(nqs, kind, N, M, Ns, iters):
    assert step(nqs, kind, N, M, Ns, kind == O.OR_CRBM, iters) < 1e-10
