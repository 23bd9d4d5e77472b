"""Measured cases of the NQS VMC step: what a user's program calls, over the sizes it calls it with.

Every case goes through the Python mirror of the C API (spin_based_neural_network_gb300.nqs).  Kinds:

  vmc     a whole sampler-driven SR step (sampling, local energies, Jacobian, solve, update) from given
          parameters: MinSR in the mixed precision, or CG-SR in FP64;
  step    one SR step on configurations the program holds: MinSR in FP64 or mixed, CG-SR, holomorphic SR;
  eloc    FP64 local energies of a batch of configurations;
  symproj log-amplitudes and gradients of a symmetry-projected complex RBM;
  sample  Metropolis batches of the FP64 Philox chains;
  batch   one step of several independent problems advanced together;
  ed      a sector Lanczos run on the kagome torus.

A step starts from the state's parameters (written into the ansatz' host mirror, as a program that
resumes from saved weights does), so repeated passes of a state do the same work.  Iterative CG-SR
solves are capped at 10 iterations, as in this repository's parity fixtures: left to run on, CG on these
ill-conditioned systems turns the last bits of its input into visible digits of the update.
"""
import math

import numpy as np
import torch

from spin_based_neural_network_gb300 import abi, nqs

HAM = {"tfim": abi.HAM_TFIM, "heis": abi.HAM_HEISENBERG, "j1j2": abi.HAM_J1_J2, "xxz": abi.HAM_XXZ,
       "kagome": abi.HAM_KAGOME_HEISENBERG}
ANSATZ = {"rbm": abi.ANSATZ_RBM, "crbm": abi.ANSATZ_COMPLEX_RBM, "mlp": abi.ANSATZ_GPU_MLP}


def listed():
    return [
        # the smallest call: CG-SR at upstream's benchmark shape (TFIM 4x4, open, 256 samples)
        {"name": "tfim4x4_rbm_cgsr", "kind": "step", "solver": "cg", "ham": "tfim", "Lx": 4, "Ly": 4, "pbc": False,
         "ansatz": "rbm", "M": 16, "Ns": 256, "mixed": False, "scale": 0.1, "shift": 1e-3, "lr": 0.01},
        # the 1-D chain workload: few long chains, everything in FP64
        {"name": "tfim16_rbm_cgsr_vmc", "kind": "vmc", "solver": "cg", "ham": "tfim", "Lx": 16, "Ly": 1, "pbc": True,
         "ansatz": "rbm", "M": 16, "Ns": 1024, "chains": 16, "decor": 16, "mixed": False, "scale": 0.01,
         "shift": 1e-3, "lr": 0.01},
        # the default MinSR call of a drop-in user: FP64, sample space, about the default 1024 samples
        {"name": "heis4x4_crbm_minsr_fp64", "kind": "step", "solver": "minsr", "ham": "heis", "Lx": 4, "Ly": 4,
         "pbc": True, "ansatz": "crbm", "M": 32, "Ns": 1000, "mixed": False, "scale": 0.1, "shift": 1e-3, "lr": 0.01},
        # the 2-D workload of the benchmark, mixed precision
        {"name": "heis4x4_crbm_minsr_vmc", "kind": "vmc", "solver": "minsr", "ham": "heis", "Lx": 4, "Ly": 4,
         "pbc": True, "ansatz": "crbm", "M": 32, "Ns": 4096, "chains": 1024, "decor": 16, "mixed": True,
         "scale": 0.01, "shift": 1e-4, "lr": 0.005},
        # the frustrated 6x6 workload: the solve in sample space at order 8192
        {"name": "j1j2_6x6_crbm_minsr_vmc", "kind": "vmc", "solver": "minsr", "ham": "j1j2", "Lx": 6, "Ly": 6,
         "pbc": True, "ansatz": "crbm", "M": 144, "Ns": 8192, "chains": 1024, "decor": 36, "mixed": True,
         "scale": 0.005, "shift": 1e-4, "lr": 0.005},
        # the largest: kagome 3x3 with the deep MLP, the solve in parameter space at order 15014
        {"name": "kagome3x3_mlp_minsr_vmc", "kind": "vmc", "solver": "minsr", "ham": "kagome", "Lx": 3, "Ly": 3,
         "pbc": True, "ansatz": "mlp", "M": 108, "Ns": 16384, "chains": 1024, "decor": 27, "mixed": True,
         "scale": 0.0, "shift": 1e-3, "lr": 0.005},
        # holomorphic SR of a p2-projected complex RBM on the 2x2 kagome torus (upstream's research run)
        {"name": "kagome2x2_p2_holo", "kind": "step", "solver": "holo", "ham": "kagome", "Lx": 2, "Ly": 2,
         "pbc": True, "ansatz": "crbm", "M": 64, "Ns": 1024, "mixed": False, "scale": 0.05, "shift": 1e-3, "lr": 0.01},
        # energy evaluation of a trained state on an odd number of configurations
        {"name": "eloc_kagome3x3_crbm", "kind": "eloc", "ham": "kagome", "Lx": 3, "Ly": 3, "pbc": True, "ansatz": "crbm",
         "M": 54, "B": 3001, "scale": 0.1},
        # projected amplitudes and gradients over the 18 translations and rotations of a 3x3 kagome torus
        {"name": "symproj_kagome3x3_p2", "kind": "symproj", "Lx": 3, "Ly": 3, "M": 40, "B": 500, "scale": 0.1},
        # plain FP64 Metropolis chains, exchange moves
        {"name": "sample_heis6x6_fp64", "kind": "sample", "Lx": 6, "Ly": 6, "ansatz": "crbm", "M": 72, "chains": 512,
         "n": 2048, "decor": 36, "exchange": True, "scale": 0.05},
        # 16 uneven instances in one launch (a quarter of the benchmark's multi-instance workload)
        {"name": "batch16_tfim_xxz", "kind": "batch", "count": 16, "pick": 2031},
        # sector Lanczos with the eigenvector, kagome 2x3 torus (2^18 states), translations
        {"name": "ed_kagome2x3", "kind": "ed", "Lx": 2, "Ly": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vmc", "vmc", "vmc", "step", "step", "step", "step", "eloc", "symproj", "sample", "batch", "ed"])
    if kind in ("step", "vmc"):
        solver = rng.choice(["minsr", "minsr", "cg"] + (["holo"] if kind == "step" else []))
        if solver == "holo":
            return {"kind": "step", "solver": "holo", "ham": "kagome", "Lx": 2, "Ly": 2, "pbc": True, "ansatz": "crbm",
                    "M": rng.randint(32, 64), "Ns": _log_int(rng, 128, 2000), "mixed": False, "scale": 0.05,
                    "shift": 1e-3, "lr": 0.01}
        ham = rng.choice(["tfim", "heis", "j1j2"]) if solver == "minsr" else "tfim"
        Lx, Ly = rng.choice([(4, 3), (4, 4), (4, 5), (6, 4), (6, 6), (10, 1), (16, 1), (20, 1)])
        if ham == "j1j2" and Ly == 1:
            Lx, Ly = 4, 4
        N = Lx * Ly
        mixed = solver == "minsr" and rng.random() < 0.6
        ansatz = rng.choice(["rbm", "crbm"]) if solver == "minsr" else "rbm"
        c = {"kind": kind, "solver": solver, "ham": ham, "Lx": Lx, "Ly": Ly, "pbc": True, "ansatz": ansatz,
             "M": N * rng.choice([1, 2, 2, 3]) + rng.choice([0, 0, 1, 5]), "mixed": mixed, "scale": 0.05,
             "shift": 1e-3, "lr": 0.01}
        if kind == "vmc":
            per = rng.choice([2, 4, 8])
            c["chains"] = _log_int(rng, 32, 1024) if mixed else _log_int(rng, 16, 256)
            c["Ns"] = c["chains"] * per
            c["decor"] = N
        else:
            c["Ns"] = _log_int(rng, 100, 6000) if mixed else _log_int(rng, 100, 2000)
        return c
    if kind == "eloc":
        ham = rng.choice(["tfim", "heis", "j1j2", "kagome"])
        Lx, Ly = rng.choice([(2, 2), (2, 3), (3, 3)] if ham == "kagome" else [(4, 4), (5, 4), (6, 6)])
        N = Lx * Ly * (3 if ham == "kagome" else 1)
        return {"kind": "eloc", "ham": ham, "Lx": Lx, "Ly": Ly, "pbc": True, "ansatz": rng.choice(["rbm", "crbm"]),
                "M": N * rng.choice([1, 2, 3]) + rng.choice([0, 1, 3]), "B": _log_int(rng, 1, 8000), "scale": 0.1}
    if kind == "symproj":
        Lx, Ly = rng.choice([(2, 2), (2, 3), (3, 3)])
        return {"kind": "symproj", "Lx": Lx, "Ly": Ly, "M": rng.randint(8, 64), "B": _log_int(rng, 1, 1000), "scale": 0.1}
    if kind == "sample":
        Lx, Ly = rng.choice([(4, 4), (4, 5), (6, 6), (12, 1)])
        N = Lx * Ly
        chains = _log_int(rng, 16, 1024)
        return {"kind": "sample", "Lx": Lx, "Ly": Ly, "ansatz": rng.choice(["rbm", "crbm"]), "M": N * rng.choice([1, 2]),
                "chains": chains, "n": chains * rng.choice([2, 4]), "decor": N, "exchange": rng.random() < 0.5,
                "scale": 0.05}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 24), "pick": rng.randrange(1 << 20)}
    Lx, Ly = rng.choice([(2, 2), (2, 3), (3, 2), (1, 5), (1, 6)])
    return {"kind": "ed", "Lx": Lx, "Ly": Ly}


# ------------------------------------------------------------------ inputs

def _sites(c):
    return c["Lx"] * c["Ly"] * (3 if c.get("ham") == "kagome" or c["kind"] in ("symproj", "ed") else 1)


def _num_params(c, N):
    M = c["M"]
    if c.get("ansatz") == "mlp":
        return M * N + M + M * M + M + 2 * M + 2
    p = N + M + M * N
    return p if c.get("ansatz") == "rbm" else 2 * p


def _spins(rng, B, N, sector):
    """Random configurations: in the smallest-|Sz| sector, or of the whole space."""
    if not sector:
        return np.where(rng.random((B, N)) < 0.5, 1, -1).astype(np.int32)
    base = np.ones(N, np.int32)
    base[:N // 2] = -1
    return rng.permuted(np.broadcast_to(base, (B, N)), axis=1)


def _sector(c):
    return c.get("ham") != "tfim"


def _marshall(c):
    return c.get("ham") in ("heis", "xxz")


def _inputs(c, seed):
    """(parameters, configurations) of a case whose program holds its configurations."""
    rng = np.random.default_rng(seed)
    N = _sites(c)
    params = rng.normal(0.0, c["scale"], size=_num_params(c, N))
    return params, _spins(rng, c["Ns"] if "Ns" in c else c["B"], N, _sector(c))


def _config(c, seed, N):
    return abi.config_defaults(
        ansatz=ANSATZ[c.get("ansatz", "crbm")], rbm_hidden_units=c["M"], width=c["M"], depth=2,
        hamiltonian=HAM[c.get("ham", "heis")], j_coupling=1.0, j2_coupling=0.5, transverse_field=1.0,
        kagome_pbc=int(c.get("pbc", True)), rng_seed=1 + seed % 1000003, num_samples=c.get("Ns", c.get("n", 1)),
        num_thermalize=4 * N, num_decorrelate=c.get("decor", 4), sr_diag_shift=c.get("shift", 1e-3),
        learning_rate=c.get("lr", 0.01), sr_cg_max_iters=10, sr_cg_tol=1e-6)


def _options(c):
    mixed = bool(c.get("mixed"))
    return dict(square_pbc=int(c.get("pbc", True)), precision=abi.PREC_MIXED if mixed else abi.PREC_FP64,
                fp32_estimator=int(mixed), refine_sweeps=8, gram_passes=3)


def _batch_specs(c, seed):
    """Uneven instances: TFIM (h in [0.5, 1.5]) and XXZ (Delta in [0.5, 2]) on chains and periodic 2-D lattices."""
    pick, rng = np.random.default_rng(c["pick"]), np.random.default_rng(seed)
    out = []
    for i in range(c["count"]):
        N = int(pick.choice([12, 16, 20, 24, 28, 32]))
        Ly = 1 if pick.integers(0, 2) == 0 else (4 if N % 8 == 0 else 2)
        alpha, Ns = int(pick.choice([1, 2])), int(pick.choice([512, 1024, 2048, 4096]))
        out.append({"xxz": i % 2 == 1, "N": N, "Lx": N // Ly, "Ly": Ly, "M": alpha * N, "Ns": Ns,
                    "h": float(rng.uniform(0.5, 1.5)), "delta": float(rng.uniform(0.5, 2.0)),
                    "seed": int(rng.integers(1, 1 << 30))})
    return out


def _prepare_batch(c, seed):
    nqs.set_options(square_pbc=1, precision=abi.PREC_MIXED, fp32_estimator=1, refine_sweeps=8, gram_passes=3)
    items, keep, views, p0 = [], [], [], []
    for sp in _batch_specs(c, seed):
        N, xxz = sp["N"], sp["xxz"]
        cfg = abi.config_defaults(ansatz=abi.ANSATZ_RBM, rbm_hidden_units=sp["M"],
                                  hamiltonian=abi.HAM_XXZ if xxz else abi.HAM_TFIM, j_coupling=1.0,
                                  j_z_coupling=sp["delta"], transverse_field=sp["h"], rng_seed=sp["seed"],
                                  num_samples=sp["Ns"], num_thermalize=4 * N, num_decorrelate=N, sr_diag_shift=1e-3,
                                  learning_rate=0.02)
        a = nqs.Ansatz(cfg, N)
        view = a.params
        view[:] = np.random.default_rng(sp["seed"]).normal(0.0, 0.1, size=a.P)
        m = nqs.Marshall(a.log_amp_fn, a.user, sp["Lx"], sp["Ly"]) if xxz else None
        fn, user = (m.log_amp_fn, m.user) if m else (a.log_amp_fn, a.user)
        o = nqs.options(num_chains=sp["Ns"] // 4, rng=abi.RNG_PHILOX,
                        move=abi.MOVE_EXCHANGE if xxz else abi.MOVE_SINGLE_FLIP, n_down=N // 2 if xxz else -1,
                        lattice_x=sp["Lx"], lattice_y=sp["Ly"], square_pbc=1, precision=abi.PREC_MIXED,
                        fp32_estimator=1)
        s = nqs.Sampler(N, cfg, fn, user, o)
        s.thermalize()
        items.append((cfg, sp["Lx"], sp["Ly"], a, s, fn if m else None, user if m else None))
        keep.append(m)
        views.append(view)
        p0.append(view.copy())
    return {"kind": "batch", "batch": nqs.Batch(items), "keep": keep, "views": views, "p0": p0}


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        return _prepare_batch(c, seed)
    N = _sites(c)
    if c["kind"] == "ed":
        perm, chars = nqs.kagome_perm(c["Lx"], c["Ly"], "translations")
        return {"kind": "ed", "c": c, "perm": perm, "chars": chars, "J": _coupling(seed)}
    opts = _options(c)
    nqs.set_options(**opts)
    cfg = _config(c, seed, N)
    st = {"kind": c["kind"], "c": c, "cfg": cfg, "N": N}
    a = st["a"] = nqs.Ansatz(cfg, N)
    view = st["view"] = a.params
    if c["kind"] in ("vmc", "sample"):
        if c.get("ansatz") != "mlp":                       # the MLP starts from its own Xavier initialisation
            view[:] = np.random.default_rng(seed).normal(0.0, c["scale"], size=a.P)
    else:
        view[:], st["spins"] = _inputs(c, seed)
    st["p0"] = view.copy()
    st["fn"], st["user"] = a.log_amp_fn, a.user
    if _marshall(c):
        st["m"] = nqs.Marshall(a.log_amp_fn, a.user, c["Lx"], c["Ly"])
        st["fn"], st["user"] = st["m"].log_amp_fn, st["m"].user
    if c["kind"] == "symproj" or c.get("solver") == "holo":
        perm, chars = nqs.kagome_perm(c["Lx"], c["Ly"], "p2")
        st["sym"] = nqs.Symproj(a.log_amp_fn, a.user, N, perm, chars)
        st["fn"], st["user"] = st["sym"].log_amp_fn, st["sym"].user
    if c["kind"] in ("vmc", "sample"):
        exchange = c["exchange"] if c["kind"] == "sample" else _sector(c)
        kw = dict(opts, num_chains=c["chains"], rng=abi.RNG_PHILOX,
                  move=abi.MOVE_EXCHANGE if exchange else abi.MOVE_SINGLE_FLIP, n_down=N // 2 if exchange else -1,
                  lattice_x=c["Lx"], lattice_y=c["Ly"], lattice_kagome=int(c.get("ham") == "kagome"))
        st["s"] = nqs.Sampler(N, cfg, st["fn"], st["user"], nqs.options(**kw))
        st["s"].thermalize()
    return st


def _coupling(seed):
    return float(np.random.default_rng(seed).uniform(0.5, 1.5))


# ------------------------------------------------------------------ one pass

def _info(i):
    return {"mean_energy": i.mean_energy, "variance_energy": i.variance_energy, "update_norm": i.update_norm,
            "acceptance_ratio": i.acceptance_ratio, "converged": i.converged}


def run(state):
    st, kind = state, state["kind"]
    if kind == "batch":
        for v, p in zip(st["views"], st["p0"]):
            v[:] = p
        infos = st["batch"].step()
        rows = [_info(i) for i in infos]
        return {"params": [v.copy() for v in st["views"]], "info": {k: np.array([r[k] for r in rows]) for k in rows[0]}}
    if kind == "ed":
        c = st["c"]
        e, vec, r = nqs.lanczos_e0_kagome_lean(c["Lx"], c["Ly"], st["J"], 1, st["perm"], st["chars"], 100, 1e-9, True)
        return {"E0": e, "vector": vec, "converged": r["converged"]}
    c = st["c"]
    if kind == "eloc":
        re, im = nqs.local_energy_batch(st["cfg"], c["Lx"], c["Ly"], st["spins"], st["fn"], st["user"], True)
        return {"re": re, "im": im}
    if kind == "symproj":
        la, ar = nqs.log_amp_batch(st["fn"], st["user"], st["spins"])
        return {"log_abs": la, "arg": ar, "gradient": nqs.symproj_gradient_batch(st["a"], st["sym"], st["spins"])}
    if kind == "sample":
        return {"spins": st["s"].batch(c["n"])}
    st["view"][:] = st["p0"]
    if kind == "vmc":
        step = nqs.sr_step_minsr if c["solver"] == "minsr" else nqs.sr_step_cg
        info = step(st["cfg"], c["Lx"], c["Ly"], st["a"], st["s"], st["fn"], st["user"])
        return {"params": st["view"].copy(), "info": _info(info)}
    gfn, guser = None, None
    if "sym" in st:
        gfn, guser = st["sym"].gradient_complex_fn, st["sym"].user
    info, E, delta = nqs.sr_step_batch(st["cfg"], c["Lx"], c["Ly"], st["a"], st["spins"],
                                       {"cg": 0, "minsr": 1, "holo": 2}[c["solver"]], st["fn"], st["user"], gfn, guser)
    return {"energies": E, "delta": delta, "params": st["view"].copy(), "info": _info(info)}


# ------------------------------------------------------------------ the work of one pass

def _bonds(c, pbc=True):
    """(nearest, diagonal) bonds of the lattice, in site indices."""
    Lx, Ly, b, d = c["Lx"], c["Ly"], [], []
    if c.get("ham") == "kagome" or c["kind"] == "ed":
        def S(x, y, k):
            return 3 * ((x % Lx) * Ly + y % Ly) + k
        for x in range(Lx):
            for y in range(Ly):
                A, B, C = S(x, y, 0), S(x, y, 1), S(x, y, 2)
                b += [(A, B), (A, C), (B, C)]
                Bm, Cm = S(x - 1, y, 1), S(x, y - 1, 2)
                b += [(A, Bm), (A, Cm), (Bm, Cm)]
        return b, d
    for x in range(Lx):
        for y in range(Ly):
            if x + 1 < Lx or (pbc and Lx > 1):
                b.append((x * Ly + y, (x + 1) % Lx * Ly + y))
            if y + 1 < Ly or (pbc and Ly > 1):
                b.append((x * Ly + y, x * Ly + (y + 1) % Ly))
    if c.get("ham") == "j1j2":
        for x in range(Lx if pbc else Lx - 1):
            for y in range(Ly if pbc else Ly - 1):
                x1, y1 = (x + 1) % Lx, (y + 1) % Ly
                d += [(x * Ly + y, x1 * Ly + y1), (x * Ly + y1, x1 * Ly + y)]
    return b, d


def _connected(c, N):
    """Connected configurations of one configuration, on average."""
    if c.get("ham") == "tfim":
        return N
    b, d = _bonds(c, c.get("pbc", True))
    return (len(b) + len(d)) / 2


def _amp_flops(c, N):
    """One amplitude ratio: an O(M) update of the hidden layer (the MLP's second layer is a dense M x M product)."""
    M = c["M"]
    return 2 * M * M + 8 * M if c.get("ansatz") == "mlp" else (16 if c.get("ansatz") == "crbm" else 4) * M


def _step_work(Ns, P, N, amp, conn, solver, sampled):
    n, k = min(Ns, P), max(Ns, P)
    if solver == "minsr":
        solve = n * (n + 1.0) * k + n ** 3 / 3.0 + 4.0 * Ns * P
    else:
        solve = 10 * 4.0 * Ns * P * (2 if solver == "holo" else 1)
    return {"bytes": 24.0 * P + (8.0 * Ns + 4.0 * Ns * N if not sampled else 8.0 * Ns),
            "flops": solve + Ns * (conn * amp + 2.0 * P) + sampled * amp}


def work(case):
    c = case
    if c["kind"] == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for sp in _batch_specs(c, 1):
            N, M = sp["N"], sp["M"]
            w = _step_work(sp["Ns"], N + M + N * M, N, 4.0 * M, N, "minsr", sp["Ns"] * N)
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    N = _sites(c)
    if c["kind"] == "ed":
        dim, iters = 2.0 ** N, 60
        return {"bytes": iters * 6 * 8.0 * dim, "flops": iters * dim * (6.0 * c["Lx"] * c["Ly"] + c["Lx"] * c["Ly"] + 8)}
    P, amp = _num_params(c, N), _amp_flops(c, N)
    if c["kind"] == "eloc":
        return {"bytes": 4.0 * c["B"] * N + 16.0 * c["B"] + 8.0 * P, "flops": c["B"] * (_connected(c, N) + 1) * amp}
    if c["kind"] == "symproj":
        G = 2 * c["Lx"] * c["Ly"]
        return {"bytes": c["B"] * (4.0 * N + 16 + 8.0 * P) + 8.0 * P, "flops": c["B"] * G * (2.0 * N * c["M"] * 2 + 3 * P)}
    if c["kind"] == "sample":
        return {"bytes": 4.0 * c["n"] * N + 8.0 * P, "flops": c["n"] * c["decor"] * float(amp)}
    G = 2 * c["Lx"] * c["Ly"] if c["solver"] == "holo" else 1
    return _step_work(c["Ns"], P, N, G * amp, _connected(c, N), c["solver"], c["Ns"] * c["decor"] if c["kind"] == "vmc" else 0)


# ------------------------------------------------------------------ the same in 64 bits, by plain torch

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tensor(a):
    return torch.as_tensor(a, dtype=torch.float64, device=_dev())


class _Rbm:
    """Real or complex RBM: log psi = a.s + sum_h log 2 cosh(b_h + W_h.s)."""

    def __init__(self, c, N, params):
        M, p = c["M"], _tensor(params)
        n = N + M + M * N
        if c.get("ansatz") != "rbm":
            p = torch.complex(p[:n], p[n:])
        self.a, self.b, self.W = p[:N], p[N:N + M], p[N + M:].reshape(M, N)

    def theta(self, s):
        return self.b + s.to(self.W.dtype) @ self.W.T

    def hidden(self, th):
        th = torch.where(th.real < 0, -th, th)             # log cosh is even
        return th + torch.log1p(torch.exp(-2 * th))

    def log_psi(self, s):
        return s.to(self.W.dtype) @ self.a + self.hidden(self.theta(s)).sum(1)

    def rows(self, s):
        """d log psi / d (a, b, W) as one row per configuration."""
        t, z = torch.tanh(self.theta(s)), s.to(self.W.dtype)
        return torch.cat([z, t, (t[:, :, None] * z[:, None, :]).reshape(len(s), -1)], 1)


def _parity(c, s):
    x = torch.arange(c["Lx"] * c["Ly"], device=s.device)
    even = ((x // c["Ly"] + x % c["Ly"]) % 2 == 0).to(s.dtype)
    return 1 - 2 * (((s < 0).to(s.dtype) * even).sum(1) % 2)


def _psi_ratio(c, amp, s, base, flip):
    """psi(s with the sites of `flip` flipped) / psi(s); base: what amp.theta or _projected gave for s."""
    s2 = s.clone()
    for u in flip:
        s2[:, u] *= -1
    if c.get("solver") == "holo":
        return _projected(c, amp, s2, base[0])[1] / base[1]
    th, hid = base
    th2, dv = th, 0.0
    for u in flip:
        th2 = th2 - 2 * s[:, u:u + 1] * amp.W[:, u]
        dv = dv - 2 * s[:, u] * amp.a[u]
    r = torch.exp(dv + (amp.hidden(th2) - hid).sum(1))
    return r * _parity(c, s2) * _parity(c, s) if _marshall(c) else r


def _p2(c):
    """Translations and the point reflection of the kagome torus as site permutations."""
    Lx, Ly, out = c["Lx"], c["Ly"], []

    def S(x, y, k):
        return 3 * ((x % Lx) * Ly + y % Ly) + k
    for dx in range(Lx):
        for dy in range(Ly):
            t, r = [0] * (3 * Lx * Ly), [0] * (3 * Lx * Ly)
            for x in range(Lx):
                for y in range(Ly):
                    for k in range(3):
                        t[S(x, y, k)] = S(x + dx, y + dy, k)
                        # the reflection about an A site takes B(x, y) to B(-x - 1, -y), C(x, y) to C(-x, -y - 1)
                        r[S(x, y, k)] = S(dx - x - (k == 1), dy - y - (k == 2), k)
            out += [t, r]
    return out


def _projected(c, amp, s, mx=None):
    """(scale, sum_g cos(arg_g) |psi(g s)| e^-scale): the group sum of the projected amplitude."""
    lp = torch.stack([amp.log_psi(s[:, g]) for g in _p2(c)])
    mx = lp.real.max(0).values if mx is None else mx
    return mx, (torch.exp(lp.real - mx) * torch.cos(lp.imag)).sum(0)


def _local_energies(c, amp, s):
    if c.get("solver") == "holo":
        base = _projected(c, amp, s)
    else:
        th = amp.theta(s)
        base = (th, amp.hidden(th))
    b, d = _bonds(c, c.get("pbc", True))
    E = torch.zeros(len(s), dtype=torch.complex128, device=s.device)
    if c["ham"] == "tfim":
        for u, v in b:
            E -= s[:, u] * s[:, v]
        for u in range(s.shape[1]):
            E -= _psi_ratio(c, amp, s, base, (u,))
        return E
    for bonds, J in ((b, 1.0), (d, 0.5)):
        for u, v in bonds:
            zz = s[:, u] * s[:, v]
            E += 0.25 * J * zz + torch.where(zz < 0, 0.5 * J * _psi_ratio(c, amp, s, base, (u, v)), 0.0)
    return E


def _symproj_rows(c, amp, s, complex_weights):
    perms = _p2(c)
    lp = torch.stack([amp.log_psi(s[:, g]) for g in perms])
    w = torch.exp(lp - lp.real.max(0).values)
    w = w if complex_weights else w.real
    w = w / w.sum(0)
    out = 0.0
    for k, g in enumerate(perms):
        o = amp.rows(s[:, g])
        out = out + w[k][:, None] * (o if complex_weights else torch.cat([o.real, -o.imag], 1))
    return out


def _cg(apply, F, iters, tol):
    x, r = torch.zeros_like(F), F.clone()
    p, rs = r.clone(), float(r @ r)
    rs0 = rs
    for _ in range(iters):
        Ap = apply(p)
        al = rs / float(p @ Ap)
        x, r = x + al * p, r - al * Ap
        new = float(r @ r)
        if new <= tol * tol * rs0:
            return x, 1
        p, rs = r + (new / rs) * p, new
    return x, 0


def _exact_step(c, seed):
    params, spins = _inputs(c, seed)
    N = _sites(c)
    s, amp = _tensor(spins), _Rbm(c, N, params)
    E, Ns = _local_energies(c, amp, s), len(spins)
    conv = 1
    if c["solver"] == "holo":
        O = _symproj_rows(c, amp, s, True)
        O = torch.cat([O, 1j * O], 1)
        m, Em = O.mean(0), E.mean()
        F = 2 * (O.mH @ E / Ns - m.conj() * Em).real

        def apply(v):
            return 2 * (O.mH @ (O @ v.to(O.dtype)) / Ns - m.conj() * (m @ v.to(O.dtype))).real + c["shift"] * v
        delta, conv = _cg(apply, F, 10, 1e-6)
    else:
        o = amp.rows(s)
        O = o if c["ansatz"] == "rbm" else torch.cat([o.real, -o.imag], 1)
        Oc, eps = O - O.mean(0), E.real - E.real.mean()
        if c["solver"] == "cg":
            delta, conv = _cg(lambda v: Oc.T @ (Oc @ v) / Ns + c["shift"] * v, Oc.T @ eps / Ns, 10, 1e-6)
        elif Ns <= O.shape[1]:
            T = Oc @ Oc.T / Ns + c["shift"] * torch.eye(Ns, dtype=torch.float64, device=Oc.device)
            delta = Oc.T @ torch.cholesky_solve(eps[:, None], torch.linalg.cholesky(T))[:, 0] / Ns
        else:
            T = Oc.T @ Oc / Ns + c["shift"] * torch.eye(O.shape[1], dtype=torch.float64, device=Oc.device)
            delta = torch.cholesky_solve((Oc.T @ eps / Ns)[:, None], torch.linalg.cholesky(T))[:, 0]
    er = E.real
    return {"energies": er.cpu().numpy(), "delta": delta.cpu().numpy(), "params": params - c["lr"] * delta.cpu().numpy(),
            "info": {"mean_energy": float(er.mean()), "variance_energy": float((er * er).mean() - er.mean() ** 2),
                     "update_norm": c["lr"] * float(delta.norm()), "acceptance_ratio": 0.0, "converged": conv}}


def _exact_ed(c, J):
    """Lowest energy of the zero-momentum sector by Lanczos on translation-averaged vectors."""
    N, Lx, Ly = _sites(c), c["Lx"], c["Ly"]
    idx = torch.arange(1 << N, device=_dev())
    bonds, _ = _bonds(c)
    anti = [((idx >> u) ^ (idx >> v)) & 1 for u, v in bonds]
    diag = sum(0.25 * (1 - 2 * a.double()) for a in anti)
    maps = []
    for dx in range(Lx):
        for dy in range(Ly):
            t = torch.zeros_like(idx)
            for x in range(Lx):
                for y in range(Ly):
                    for k in range(3):
                        t |= ((idx >> (3 * (x * Ly + y) + k)) & 1) << (3 * ((x + dx) % Lx * Ly + (y + dy) % Ly) + k)
            maps.append(t)

    def mul(v):
        w = diag * v
        for (u, x), a in zip(bonds, anti):
            w += torch.where(a == 1, 0.5 * v[idx ^ ((1 << u) | (1 << x))], 0.0)
        return sum(w[t] for t in maps) / len(maps)
    v = _tensor(np.random.default_rng(0).random(1 << N) - 0.5)
    v = sum(v[t] for t in maps)
    v /= v.norm()
    prev, beta, al, be = torch.zeros_like(v), 0.0, [], []
    for _ in range(90):
        w = mul(v) - beta * prev
        al.append(float(w @ v))
        w -= al[-1] * v
        beta = float(w.norm())
        if beta < 1e-12:
            break
        be.append(beta)
        prev, v = v, w / beta
    T = np.diag(al) + np.diag(be[:len(al) - 1], 1) + np.diag(be[:len(al) - 1], -1)
    return J * float(np.linalg.eigvalsh(T)[0])


def exact(case, seed):
    c = case
    if c["kind"] in ("vmc", "sample", "batch"):            # their configurations come out of the sampler
        return None
    if c["kind"] == "step":
        return _exact_step(c, seed)
    if c["kind"] == "ed":
        return {"E0": _exact_ed(c, _coupling(seed)), "vector": None, "converged": None}
    params, spins = _inputs(c, seed)
    amp, s = _Rbm(c, _sites(c), params), _tensor(spins)
    if c["kind"] == "eloc":
        E = _local_energies(c, amp, s)
        return {"re": E.real.cpu().numpy(), "im": E.imag.cpu().numpy() if c["ansatz"] == "crbm" else None}
    mx, z = _projected(c, amp, s)
    la = torch.log(z.abs()) + mx - 0.5 * math.log(2 * c["Lx"] * c["Ly"])
    arg = (z < 0).double() * math.pi
    return {"log_abs": la.cpu().numpy(), "arg": arg.cpu().numpy(),
            "gradient": _symproj_rows(c, amp, s, False).cpu().numpy()}
