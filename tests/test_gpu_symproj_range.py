"""Symmetry-projected RBM / complex RBM over the whole range of the weights: local energies of peaked states
whose products stay in range.  The reference is the definition in extended precision (long double)."""
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


class Extended:
    """sum_g chi_g cos(arg_g) |psi(g s)| of an RBM / complex RBM in long double, one scale per set of states."""

    def __init__(self, kind, N, M, params, perm, chars):
        p = params.astype(np.longdouble)
        n = N + M + M * N
        p = p[:n] + 1j * p[n:] if kind == O.OR_CRBM else p.astype(np.clongdouble)
        self.a, self.b, self.W, self.perm, self.chars = p[:N], p[N:N + M], p[N + M:].reshape(M, N), perm, chars

    def log_psi(self, s):
        """[G] log psi(g s) of one configuration."""
        gs = s[self.perm].astype(np.longdouble)
        th = self.b + gs @ self.W.T
        th = np.where(th.real < 0, -th, th)
        return gs @ self.a + np.sum(th + np.log1p(np.exp(-2 * th)), axis=1)

    def project(self, s, scale):
        """(projected psi, sum_g |terms|), both times exp(-scale)."""
        l = self.log_psi(s)
        m = self.chars * np.exp(l.real - scale)
        return np.sum(m * np.cos(l.imag)), np.sum(np.abs(m))

    def energy(self, bonds, s):
        """(E, sum of |terms| of E, |psi| over the sum of its terms' moduli) for H = sum S_u.S_v."""
        scale = self.log_psi(s).real.max()
        psi, mod = self.project(s, scale)
        e, den = np.longdouble(0), np.longdouble(1)
        for u, v in bonds:
            e += np.longdouble(s[u] * s[v]) / 4
            if s[u] != s[v]:
                t = s.copy()
                t[u], t[v] = -t[u], -t[v]
                x = self.project(t, scale)[0] / psi / 2
                e, den = e + x, den + abs(x)
        return float(e), float(den), float(abs(psi) / mod)


def setup(nqs, kind, M, params, irrep="A1"):
    from spin_based_neural_network_gb300 import abi
    perm, chars = nqs.kagome_perm(2, 2, "p6m", irrep)
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=M, hamiltonian=abi.HAM_KAGOME_HEISENBERG, kagome_pbc=1)
    a = nqs.Ansatz(cfg, 12)
    a.params[:] = params(a.P)
    sym = nqs.Symproj(a.log_amp_fn, a.user, 12, perm, chars)
    perm = np.asarray(perm).reshape(-1, 12)
    return cfg, a, sym, Extended(kind, 12, M, a.params.copy(), perm, np.asarray(chars, np.longdouble))


def configurations(B, seed):
    return np.where(np.random.default_rng(seed).random((B, 12)) < 0.5, 1, -1).astype(np.int32)


# ratios of |log psi| of a few 10^2 and the theta of 10 units: 1e-13, over the 1e-3 that a projected sum may
# cancel to; the logarithms' path has the same
@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("std", [0.1, 1.0, 2.0, 5.0])
def test_energies_of_peaked_states(nqs, kind, std):
    cfg, a, sym, ext = setup(nqs, kind, 10, lambda P: np.random.default_rng(7).normal(0.0, std, size=P))
    spins = configurations(24, 3)
    e = nqs.local_energy_batch(cfg, 2, 2, spins, sym.log_amp_fn, sym.user)
    bonds = O.bonds(O.ham(6, 2, 2, kagome_pbc=1))
    seen = 0
    for k, s in enumerate(spins):
        want, den, cond = ext.energy(bonds, s)
        if cond > 1e-3:
            seen += 1
            assert abs(e[k] - want) < 1e-9 * den, (k, e[k], want)
    assert seen > 8
