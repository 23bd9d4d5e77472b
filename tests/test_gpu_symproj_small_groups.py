"""Projections of one to four elements, on both sides of the number from which a kernel of their own takes them:
log-amplitudes and gradients against the oracle."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_symproj_prod import rel, setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nqs():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import nqs as N
    N.set_options()
    return N


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("G", [1, 2, 3, 4])
@pytest.mark.parametrize("M", [1, 40])
def test_few_elements(nqs, kind, G, M):
    rng = np.random.default_rng(10 * G + M)
    perm = np.stack([rng.permutation(12) for _ in range(G)]).astype(np.int32)
    cfg, a, sym, fn, user, keep, amp = setup(nqs, kind, 12, M, perm, np.array([1.0, 0.5, 1.0, 0.7])[:G], 0.1, G, ("in", "out"),
                                             hamiltonian=6, kagome_pbc=1)
    spins = np.where(rng.random((37, 12)) < 0.5, 1, -1).astype(np.int32)
    la, ar = nqs.log_amp_batch(fn, user, spins)
    lo, ao = O.log_amp(amp, spins)
    full = O.log_amp(O.Amp(kind, 12, M, a.params.copy()), spins)[0]
    good = lo > full - np.log(1e4)                           # a node loses the digits that cancel
    assert good.sum() > 10
    assert rel(la[good], lo[good]) < 1e-11
    assert np.max(np.abs(np.angle(np.exp(1j * (ar[good] - ao[good]))))) < 1e-12
    inner = O.Amp(kind, 12, M, a.params.copy(), [("symproj", perm.reshape(-1), np.array([1.0, 0.5, 1.0, 0.7])[:G]),
                                                 ("marshall", 3, 4)])
    g = nqs.symproj_gradient_batch(a, sym, spins)
    assert rel(g[good], O.symproj_gradient(inner, spins)[good]) < 1e-8
    if kind == O.OR_CRBM:
        gr, gi = nqs.symproj_gradient_complex_batch(a, sym, spins)
        og = O.symproj_gradient_complex(inner, spins)
        assert rel(gr[good], og[0][good]) < 1e-8 and rel(gi[good], og[1][good]) < 1e-8
