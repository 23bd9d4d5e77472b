"""FP64 local energies in product form at the edges of their tiles: hidden widths around the
lane-group boundaries (8 / 16 / 32 lanes a configuration), single configurations, both move sets,
and weights whose products leave a double's range (evaluated through the logarithms).  The
reference is the definition in extended precision (long double), on the oracle's bonds: at 192
hidden units the oracle's own double-precision sums of log cosh are 1e-12 off."""
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


def energies(nqs, kind, M, ham, Lx, Ly, scale, B, seed):
    from spin_based_neural_network_gb300 import abi
    N = Lx * Ly
    rng = np.random.default_rng(seed)
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=M, hamiltonian=ham, j2_coupling=0.5, j_z_coupling=1.3,
                              transverse_field=0.8)
    a = nqs.Ansatz(cfg, N)
    a.params[:] = rng.normal(0.0, scale, size=a.P)
    m = nqs.Marshall(a.log_amp_fn, a.user, Lx, Ly)
    spins = np.where(rng.random((B, N)) < 0.5, 1, -1).astype(np.int32)
    nqs.set_options(square_pbc=1)
    try:
        re, im = nqs.local_energy_batch(cfg, Lx, Ly, spins, m.log_amp_fn, m.user, complex_out=True)
    finally:
        nqs.set_options()
    h = O.ham(ham, Lx, Ly, pbc=1, J2=0.5, Jz=1.3, Gamma=0.8)
    return np.array(re) + 1j * np.array(im), extended(kind, N, M, a.params.copy(), h, spins, Lx, Ly)


def extended(kind, N, M, params, h, spins, Lx, Ly):
    """Local energies with the Marshall sign, in long double."""
    p = params.astype(np.longdouble)
    n = N + M + M * N
    if kind == O.OR_CRBM:
        p = p[:n] + 1j * p[n:]
    va, vb, W = p[:N], p[N:N + M], p[N + M:].reshape(M, N)
    even = np.array([(i // Ly + i % Ly) % 2 == 0 for i in range(N)])
    out = np.zeros(len(spins), np.clongdouble)
    b1 = [tuple(b) for b in O.bonds(h)]
    b2 = []
    if h.ham == 2:
        for x in range(Lx):
            for y in range(Ly if Ly > 1 else 0):
                x1, y1 = (x + 1) % Lx, (y + 1) % Ly
                b2 += [(x * Ly + y, x1 * Ly + y1), (x * Ly + y1, x1 * Ly + y)]
    for k, s in enumerate(spins.astype(np.longdouble)):
        th = vb + W @ s

        def ratio(*flip):
            t, w, d = s.copy(), np.longdouble(0), th
            for u in flip:
                t[u], w, d = -t[u], w - 2 * va[u] * s[u], d - 2 * s[u] * W[:, u]
            sign = (-1) ** int(np.sum((t < 0) & even) + np.sum((s < 0) & even))
            return sign * np.exp(w) * np.prod(np.cosh(d) / np.cosh(th))
        if h.ham == 0:
            out[k] = -sum(s[u] * s[v] for u, v in b1) - np.longdouble(h.Gamma) * sum(ratio(u) for u in range(N))
            continue
        jz = h.Jz if h.ham == 4 else h.J
        for bonds, z, x in ((b1, jz, h.J), (b2, h.J2, h.J2)):
            for u, v in bonds:
                out[k] += np.longdouble(z) / 4 * s[u] * s[v]
                if s[u] != s[v]:
                    out[k] += np.longdouble(x) / 2 * ratio(u, v)
    return out


@pytest.mark.parametrize("M", [1, 16, 17, 64, 65, 96, 128, 129, 192, 256])
@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
def test_widths(nqs, kind, M):
    # the parity bar of the FP64 path: 1e-12 of max(|E|, 1)
    for ham, Lx, Ly, B in ((0, 5, 1, 1), (2, 4, 3, 33), (4, 7, 1, 3), (2, 6, 6, 5)):
        e, r = energies(nqs, kind, M, ham, Lx, Ly, 0.15, B, 10 * M + ham)
        assert np.max(np.abs(e - r) / np.maximum(np.abs(r), 1.0)) < 1e-12, (ham, Lx, Ly)


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
def test_weights_out_of_range(nqs, kind):
    # through the logarithms: |log psi| reaches a few 10^3, and exp(log ratio) carries about
    # 8 x 2^-53 x 4e3 = 4e-12 relative
    for ham in (0, 2):
        e, r = energies(nqs, kind, 40, ham, 4, 3, 8.0, 40, 3)
        assert np.all(np.isfinite(r.real))
        assert np.max(np.abs(e - r) / np.maximum(np.abs(r), 1.0)) < 1e-11


def test_non_finite_parameters(nqs):
    """Infinite or NaN parameters give NaN energies; only an infinite visible bias does not, since
    flipping its spin away from it has ratio 0 and no other flip involves it."""
    from spin_based_neural_network_gb300 import abi
    cfg = abi.config_defaults(ansatz=abi.ANSATZ_RBM, rbm_hidden_units=8, hamiltonian=abi.HAM_TFIM)
    spins = np.ones((2, 6), np.int32)
    for k in (2, 7, 20):                     # a visible bias, a hidden bias, a weight
        for bad in (np.inf, np.nan):
            a = nqs.Ansatz(cfg, 6)
            a.params[k] = bad
            e = nqs.local_energy_batch(cfg, 6, 1, spins, a.log_amp_fn, a.user)
            assert (np.isfinite(e) if k == 2 and bad == np.inf else np.isnan(e)).all()
