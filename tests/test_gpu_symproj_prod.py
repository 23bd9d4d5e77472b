"""Symmetry-projected RBM / complex RBM in product form: log-amplitudes, gradients and local energies
against the oracle for groups of 4 to 48 elements with real characters of both signs, Marshall layers
inside and outside, hidden widths around the lane groups, maps that are not one to one, and weights
beyond the range of the products."""
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


def setup(nqs, kind, N, M, perm, chars, scale, seed, marshall=(), **cfg_kw):
    from spin_based_neural_network_gb300 import abi
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=M, **cfg_kw)
    a = nqs.Ansatz(cfg, N)
    a.params[:] = np.random.default_rng(seed).normal(0.0, scale, size=a.P)
    fn, user, keep, layers = a.log_amp_fn, a.user, [a], []
    if "in" in marshall:
        keep.append(nqs.Marshall(fn, user, 3, N // 3))
        fn, user = keep[-1].log_amp_fn, keep[-1].user
        layers.insert(0, ("marshall", 3, N // 3))
    sym = nqs.Symproj(fn, user, N, perm, chars)
    keep.append(sym)
    fn, user = sym.log_amp_fn, sym.user
    layers.insert(0, ("symproj", np.asarray(perm).reshape(-1), chars))
    if "out" in marshall:
        keep.append(nqs.Marshall(fn, user, 3, N // 3))
        fn, user = keep[-1].log_amp_fn, keep[-1].user
        layers.insert(0, ("marshall", 3, N // 3))
    return cfg, a, sym, fn, user, keep, O.Amp(kind, N, M, a.params.copy(), layers)


def rel(x, y):
    return float(np.max(np.abs(x - y) / np.maximum(np.abs(y), 1.0)))


def kagome(nqs, group, irrep="A1"):
    return nqs.kagome_perm(2, 2, group, irrep)


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("M", [1, 9, 16, 17, 33, 64, 65, 128, 200])
@pytest.mark.parametrize("group,irrep,marshall", [("translations", "A1", ()), ("p2", "A1", ("in", "out")),
                                                  ("p6m", "B1", ("in",)), ("p6m", "E2", ())])
def test_against_oracle(nqs, kind, M, group, irrep, marshall):
    perm, chars = kagome(nqs, group, irrep)
    cfg, a, sym, fn, user, keep, amp = setup(nqs, kind, 12, M, perm, chars, 0.12, M, marshall, hamiltonian=6,
                                             kagome_pbc=1)
    spins = np.where(np.random.default_rng(M).random((13, 12)) < 0.5, 1, -1).astype(np.int32)
    la, ar = nqs.log_amp_batch(fn, user, spins)
    lo, ao = O.log_amp(amp, spins)
    # a node of the projected state loses the digits that cancel in its group sum: log|psi| below
    # the largest element by ln(1e4) is left out
    full = O.log_amp(O.Amp(kind, 12, M, a.params.copy()), spins)[0]
    good = lo > full - np.log(1e4)
    assert good.any() or irrep != "A1"
    if good.any():
        assert rel(la[good], lo[good]) < 1e-11
        assert np.max(np.abs(np.angle(np.exp(1j * (ar[good] - ao[good]))))) < 1e-12
    e = nqs.local_energy_batch(cfg, 2, 2, spins, fn, user)
    eo = O.local_energy(O.ham(6, 2, 2, kagome_pbc=1), amp, spins)
    if good.any():
        assert np.max(np.abs(e - eo)[good] / np.maximum(np.abs(eo[good]), 1.0)) < 1e-8    # 1e-12 over the 1e4 of a node
    if "out" not in marshall and good.any():
        g = nqs.symproj_gradient_batch(a, sym, spins)
        assert rel(g[good], O.symproj_gradient(amp, spins)[good]) < 1e-8
        if kind == O.OR_CRBM:
            gr, gi = nqs.symproj_gradient_complex_batch(a, sym, spins)
            og = O.symproj_gradient_complex(amp, spins)
            den = np.maximum(np.abs(og[0]), 1.0), np.maximum(np.abs(og[1]), 1.0)
            assert np.max((np.abs(gr - og[0]) / den[0])[good]) < 1e-8
            assert np.max((np.abs(gi - og[1]) / den[1])[good]) < 1e-8


@pytest.mark.parametrize("kind", [O.OR_RBM, O.OR_CRBM])
@pytest.mark.parametrize("ham", [0, 1, 2])
def test_square_translations_all_moves(nqs, kind, ham):
    from spin_based_neural_network_gb300 import abi
    N, M = 12, 20
    cfg = abi.config_defaults(ansatz=kind, rbm_hidden_units=M, hamiltonian=ham, j2_coupling=0.4, transverse_field=0.7)
    a = nqs.Ansatz(cfg, N)
    a.params[:] = np.random.default_rng(4).normal(0.0, 0.05, size=a.P)
    t = nqs.Translation(a.log_amp_fn, a.user, 4, 3)
    spins = np.where(np.random.default_rng(5).random((21, N)) < 0.5, 1, -1).astype(np.int32)
    perm = np.array([[((x + tx) % 4) * 3 + (y + ty) % 3 for x in range(4) for y in range(3)]
                     for tx in range(4) for ty in range(3)])
    amp = O.Amp(kind, N, M, a.params.copy(), [("symproj", perm.reshape(-1), np.ones(12))])
    e = nqs.local_energy_batch(cfg, 4, 3, spins, t.log_amp_fn, t.user)
    assert rel(e, O.local_energy(O.ham(ham, 4, 3, J2=0.4, Gamma=0.7), amp, spins)) < 1e-12


def test_maps_that_are_not_one_to_one(nqs):
    rng = np.random.default_rng(8)
    perm = np.stack([np.arange(12), rng.integers(0, 12, 12), rng.permutation(12)]).astype(np.int32)
    cfg, a, sym, fn, user, keep, amp = setup(nqs, O.OR_CRBM, 12, 10, perm, np.array([1.0, 0.5, 1.0]), 0.1, 2, (),
                                             hamiltonian=6, kagome_pbc=1)
    spins = np.where(rng.random((9, 12)) < 0.5, 1, -1).astype(np.int32)
    e = nqs.local_energy_batch(cfg, 2, 2, spins, fn, user)
    assert rel(e, O.local_energy(O.ham(6, 2, 2, kagome_pbc=1), amp, spins)) < 1e-12


@pytest.mark.parametrize("kind", [O.OR_RBM])
def test_weights_out_of_range(nqs, kind):
    perm, chars = kagome(nqs, "translations")
    cfg, a, sym, fn, user, keep, amp = setup(nqs, kind, 12, 40, perm, chars, 8.0, 3, (), hamiltonian=6, kagome_pbc=1)
    spins = np.where(np.random.default_rng(3).random((15, 12)) < 0.5, 1, -1).astype(np.int32)
    e = nqs.local_energy_batch(cfg, 2, 2, spins, fn, user)
    eo = O.local_energy(O.ham(6, 2, 2, kagome_pbc=1), amp, spins)
    assert np.max(np.abs(e - eo) / np.maximum(np.abs(eo), 1.0)) < 1e-11       # |log psi| of a few 10^3, 8 roundings
