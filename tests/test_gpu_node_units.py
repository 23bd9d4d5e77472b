"""Complex RBM whose hidden units stand near their nodes (hidden biases i pi / 2: cosh acts as i sinh), so that
the product of their |1 + exp(-2 theta)| falls to 1e-370, with and without a symmetry projection.  The reference
is the definition in extended precision (long double); gradients against the oracle's sums of logarithms."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_symproj_range import Extended, configurations

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nqs():
    import spin_based_neural_network_gb300 as pkg
    pkg.build()
    from spin_based_neural_network_gb300 import nqs as N
    N.set_options()
    return N


def ansatz(nqs, M, N=12):
    from spin_based_neural_network_gb300 import abi
    cfg = abi.config_defaults(ansatz=O.OR_CRBM, rbm_hidden_units=M, hamiltonian=abi.HAM_KAGOME_HEISENBERG, kagome_pbc=1)
    a = nqs.Ansatz(cfg, N)
    a.params[:] = np.random.default_rng(M).normal(0.0, 0.005, size=a.P)
    a.params[a.P // 2 + N:a.P // 2 + N + M] = np.pi / 2
    return cfg, a


# theta' of 0.005 to 0.05 beside pi / 2: 2e-14 a unit, 5e-12 for 256, over the 1e-3 that a projected sum may cancel to
@pytest.mark.parametrize("M", [12, 64, 144, 256])
def test_projected(nqs, M):
    perm, chars = nqs.kagome_perm(2, 2, "p6m", "A1")
    cfg, a = ansatz(nqs, M)
    sym = nqs.Symproj(a.log_amp_fn, a.user, 12, perm, chars)
    perm = np.asarray(perm).reshape(-1, 12)
    ext = Extended(O.OR_CRBM, 12, M, a.params.copy(), perm, np.asarray(chars, np.longdouble))
    amp = O.Amp(O.OR_CRBM, 12, M, a.params.copy(), [("symproj", perm.reshape(-1), np.asarray(chars, float))])
    spins = configurations(40, M)
    la, ar = nqs.log_amp_batch(sym.log_amp_fn, sym.user, spins)
    e = nqs.local_energy_batch(cfg, 2, 2, spins, sym.log_amp_fn, sym.user)
    g, og = nqs.symproj_gradient_batch(a, sym, spins), O.symproj_gradient(amp, spins)
    c, oc = nqs.symproj_gradient_complex_batch(a, sym, spins), O.symproj_gradient_complex(amp, spins)
    bonds = O.bonds(O.ham(6, 2, 2, kagome_pbc=1))
    seen = 0
    for k, s in enumerate(spins):
        scale = ext.log_psi(s).real.max()
        psi, mod = ext.project(s, scale)
        if not abs(psi) > 1e-3 * mod:
            continue
        seen += 1
        want, den, _ = ext.energy(bonds, s)
        assert abs(la[k] - float(np.log(abs(psi)) + scale - np.log(np.longdouble(len(chars))) / 2)) < 1e-8
        assert abs(np.cos(ar[k]) - float(np.sign(psi))) < 1e-8
        assert abs(e[k] - want) < 1e-8 * den
        for x, y in ((g, og), (c[0], oc[0]), (c[1], oc[1])):
            assert np.max(np.abs(x[k] - y[k])) < 1e-8 * max(np.max(np.abs(y[k])), 1.0)
    assert seen > 8


@pytest.mark.parametrize("M", [12, 64, 144, 256])
def test_unprojected(nqs, M):
    cfg, a = ansatz(nqs, M)
    ext = Extended(O.OR_CRBM, 12, M, a.params.copy(), np.arange(12)[None, :], np.ones(1, np.longdouble))
    spins = configurations(40, M)
    re, im = nqs.local_energy_batch(cfg, 2, 2, spins, a.log_amp_fn, a.user, complex_out=True)
    for k, s in enumerate(spins):
        l0, want, den = ext.log_psi(s)[0], 0.0, 1.0
        for u, v in O.bonds(O.ham(6, 2, 2, kagome_pbc=1)):
            want += np.longdouble(s[u] * s[v]) / 4
            if s[u] != s[v]:
                t = s.copy()
                t[u], t[v] = -t[u], -t[v]
                x = np.exp(ext.log_psi(t)[0] - l0) / 2
                want, den = want + x, den + abs(x)
        assert abs(re[k] + 1j * im[k] - complex(want)) < 5e-12 * den
