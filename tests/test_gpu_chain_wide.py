"""FP64 Philox chains whose weights leave the product form's range in every unit, over the widths of a lane: the
oracle's chains sample for sample, at O(M) a proposal (through log cosh of the units, not the whole amplitude)."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_chain_range import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nqs():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import nqs as N
    N.set_options()
    return N


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 70, 130, 256])
@pytest.mark.parametrize("exchange", [False, True])
def test_weights_out_of_range(nqs, kind, M, exchange):
    def fill(p):
        p *= 600.0 / np.sqrt(M)                            # standard deviation 30 over the root of M, and
        p[16] = 320.0                                      # the first hidden bias: past the bound of |theta|
    nqs.profile(True)
    nqs.profile_reset()
    try:
        compare(nqs, kind, 4, 4, M, fill, exchange)
        names = set(nqs.profile_read())
    finally:
        nqs.profile(False)
    assert "sampler" in names and "sampler_generic" not in names
