"""The work a user of this framework has it do, as cases that can be timed.

Every case is one pass through the public Python interface over the C ABI
(``Chain`` and its methods), the way a host program drives it:

* ``bond``     one TwoSiteOp with the bond's tensors handed in by the host, as a
               Fortran host that keeps its own chain calls it
* ``quench``   Trotter steps from a product state: the start of every run, where
               the bonds are unsaturated and the calls small
* ``ring``     the same with periodic boundaries (swaps, one bond after another)
* ``sweep``    one batched sweep over the odd bonds of a saturated chain, the
               regime that most of a long run is spent in; in plain FP64, in the
               double-float form and in the mixed form
* ``step``     whole Trotter steps (2nd order or Forest-Ruth) of a saturated chain
* ``nc``       a Trotter step of a saturated number-conserving chain
* ``measure``  the observables of a chain that is on the device

A pass uploads its chain from pinned host memory first (a pass on the same state
is therefore the same work again), and returns what such a program reads back:
every Lambda, the one-site density matrix of every site, the kept weight, and
two-site density matrices where the case is about them.  Gammas are not
returned: they are defined up to a gauge (the phases of the singular vectors),
which the density matrices do not see.

A case's numbers: L sites, local dimension d, bond dimension chi, time step dt,
Trotter ``order`` 2 or 5 (Forest-Ruth), ``steps``; ``svd`` is the form of the SVD
(fp64, df, mixed: see FORMS).
"""
import math

import numpy as np
import torch

import __graft_entry__

# form -> (svd_mode, theta form): plain FP64; double-float; the mixed form
# (randomized route, Theta on the tensor cores; number-conserving chains:
# double-float block SVDs and Theta's block products on the tensor cores)
FORMS = {"fp64": (0, 0), "df": (5, 0), "mixed": (6, 107), "nc_mixed": (5, 107)}


def _pkg():
    return __graft_entry__.load_package()


def listed():
    return [
        # a Fortran host calls TwoSiteOp on its own arrays, small chain: the smallest call
        {"name": "bond_d2_chi16", "kind": "bond", "d": 2, "chi": 16, "dt": 0.05},
        # spin-1/2 XXZ chain from the Neel state, the CPU-sized configuration (L=32, chi=32)
        {"name": "xxz_quench_chi32", "kind": "quench", "model": "xxz", "L": 32, "d": 2, "chi": 32, "dt": 0.01,
         "order": 2, "steps": 12},
        # periodic ring, odd length and odd chi: swaps, one small bond at a time
        {"name": "xxz_ring_L13_chi45", "kind": "ring", "model": "xxz", "L": 13, "d": 2, "chi": 45, "dt": 0.05,
         "order": 2, "steps": 2},
        # the headline run's first steps: Bose-Hubbard L=64, d=5, chi=128 from the perturbed Mott state
        {"name": "bose_quench_chi128", "kind": "quench", "model": "bose", "L": 64, "d": 5, "chi": 128, "dt": 0.005,
         "order": 2, "steps": 8},
        # spin-1 chain, Forest-Ruth step at a ragged size (Theta 270 x 270)
        {"name": "spin1_forest_ruth_chi90", "kind": "step", "model": "spin1", "L": 20, "d": 3, "chi": 90, "dt": 0.01,
         "order": 5, "steps": 1, "svd": "fp64"},
        # the headline run once saturated: 32 bonds of a 640 x 640 Theta, plain FP64
        {"name": "bose_sweep_chi128", "kind": "sweep", "model": "bose", "L": 64, "d": 5, "chi": 128, "dt": 0.005,
         "svd": "fp64"},
        # the same bonds in the mixed form
        {"name": "bose_sweep_chi128_mixed", "kind": "sweep", "model": "bose", "L": 64, "d": 5, "chi": 128,
         "dt": 0.005, "svd": "mixed"},
        # Fermi-Hubbard chi=256, double-float form: 1024 x 1024 Thetas
        {"name": "fermi_sweep_chi256_df", "kind": "sweep", "model": "fermi", "L": 24, "d": 4, "chi": 256, "dt": 0.01,
         "svd": "df"},
        # the largest Theta of the configured runs (2560 x 2560), mixed form
        {"name": "bose_sweep_chi512_mixed", "kind": "sweep", "model": "bose", "L": 16, "d": 5, "chi": 512,
         "dt": 0.005, "svd": "mixed"},
        # number-conserving Bose-Hubbard, plain FP64
        {"name": "nc_step_chi256", "kind": "nc", "model": "bose", "L": 32, "d": 5, "chi": 256, "dt": 0.01,
         "svd": "fp64"},
        # number-conserving at the configured chi=512, mixed form
        {"name": "nc_step_chi512_mixed", "kind": "nc", "model": "bose", "L": 16, "d": 5, "chi": 512, "dt": 0.01,
         "svd": "nc_mixed"},
        # densities, bond energies, entropies and the overlap of a saturated chain
        {"name": "measure_chi128", "kind": "measure", "model": "bose", "L": 64, "d": 5, "chi": 128},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# the largest work one drawn case may have: bonds x (d chi)^3 of the saturated sweep
_MOST = 32 * 640 ** 3


def draw(rng):
    kind = rng.choice(["bond", "quench", "ring", "step", "sweep", "sweep", "nc", "measure"])
    if kind == "bond":
        return {"kind": "bond", "d": rng.choice([2, 3, 4, 5]), "chi": _logint(rng, 7, 50), "dt": 0.05}
    if kind == "ring":
        return {"kind": "ring", "model": "xxz", "L": rng.randint(7, 16), "d": 2, "chi": _logint(rng, 16, 64),
                "dt": 0.05, "order": 2, "steps": rng.randint(1, 3)}
    model = rng.choice(["xxz", "spin1", "fermi", "bose"])
    d = {"xxz": 2, "spin1": 3, "fermi": 4, "bose": rng.choice([3, 4, 5])}[model]
    if kind == "quench":
        return {"kind": "quench", "model": model, "L": rng.randint(8, 64), "d": d, "chi": _logint(rng, 16, 128),
                "dt": rng.choice([0.005, 0.01]), "order": rng.choice([2, 2, 5]), "steps": rng.randint(2, 6)}
    if kind == "step":
        chi = _logint(rng, 24, 360 // d)
        return {"kind": "step", "model": model, "L": rng.randint(6, 32), "d": d, "chi": chi, "dt": 0.01,
                "order": rng.choice([2, 5]), "steps": 1, "svd": rng.choice(["fp64", "fp64", "df"])}
    if kind == "sweep":
        svd = rng.choice(["fp64", "df", "mixed"])
        chi = _logint(rng, 96 if svd == "mixed" else 48, 300)
        most = _MOST * (4 if svd == "mixed" else 1)
        bonds = max(1, min(32, int(most / (d * chi) ** 3)))
        if bonds * (d * chi) ** 3 > most:
            d, model = 3, "spin1"
            bonds = max(1, min(32, int(most / (d * chi) ** 3)))
        return {"kind": "sweep", "model": model, "L": 2 * rng.randint(max(1, bonds // 3), bonds), "d": d, "chi": chi,
                "dt": rng.choice([0.005, 0.01]), "svd": svd}
    if kind == "nc":
        d = rng.choice([3, 4, 5])
        return {"kind": "nc", "model": "bose", "L": rng.randint(8, 24), "d": d, "chi": _logint(rng, 64, 300),
                "dt": 0.01, "svd": rng.choice(["fp64", "nc_mixed"])}
    return {"kind": "measure", "model": model, "L": rng.randint(8, 64), "d": d, "chi": _logint(rng, 16, 160)}


# ---------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------
def _hamiltonian(case, seed):
    H = _pkg().hamiltonians
    L, d, model = case["L"], case["d"], case["model"]
    rng = np.random.default_rng([seed, 77])
    if model == "xxz":
        return H.heisenberg(L, 1.0, 1.0, 1.0)
    if model == "spin1":
        return H.spin1_xxz_anisotropy(L, 1.0, 1.0, rng.uniform(-0.5, 0.5, L))
    if model == "fermi":
        return H.fermi_hubbard(L, 1.0, 4.0)
    if case["kind"] == "nc":
        return H.bose_hubbard(L, d, 1.0, rng.uniform(1.0, 3.0, L))
    return H.bose_hubbard(L, d, 1.0, 2.0)


def _gates(case, seed):
    H = _pkg().hamiltonians
    if case["kind"] == "ring":
        h = _hamiltonian(dict(case, L=case["L"] + 1), seed)  # L bond terms, the last one the edge bond
        return H.construct_propagators(h, case["dt"], case["order"], boundary="P")
    return H.construct_propagators(_hamiltonian(case, seed), case["dt"], case.get("order", 2))


# ---------------------------------------------------------------------------
# states, in pinned host memory: Gammas (chi, d, chi) Fortran-ordered, Lambdas
# ---------------------------------------------------------------------------
def _pinned(x):
    """A (b, i, a) tensor as the Fortran-ordered (a, i, b) array a host program holds."""
    out = torch.empty(x.shape, dtype=x.dtype, pin_memory=torch.cuda.is_available())
    out.copy_(x)
    return out.numpy().T


def _generator(seed, salt):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return torch.Generator(device=dev).manual_seed(int(seed) * 1000003 + salt), dev


def _randn(shape, g, dev):
    return torch.complex(torch.randn(shape, generator=g, device=dev, dtype=torch.float64),
                         torch.randn(shape, generator=g, device=dev, dtype=torch.float64))


def _product_state(case, seed):
    """The product state a quench starts from, with a seeded complex perturbation
    of amplitude 1e-3 on every Gamma entry, each site renormalised."""
    L, d, chi, model = case["L"], case["d"], case["chi"], case["model"]
    c = np.zeros((d, L))
    for i in range(L):
        c[{"xxz": i % 2, "spin1": 2 * (i % 2), "fermi": 1 + i % 2, "bose": 1}[model], i] = 1.0
    g, dev = _generator(seed, 1)
    gam, lam = [], []
    for i in range(L):
        x = 1e-3 * _randn((chi, d, chi), g, dev)
        x[0, :, 0] += torch.as_tensor(c[:, i], device=dev)
        x[0, :, 0] /= torch.linalg.vector_norm(x[0, :, 0])
        gam.append(_pinned(x))
    for _ in range(L + 1):
        v = np.zeros(chi)
        v[0] = 1.0
        lam.append(v)
    return gam, lam


def _spectrum(chi, n=None):
    """A saturated bond's Schmidt values, lambda_k ~ exp(-12 k / chi)."""
    v = np.zeros(chi)
    k = np.arange(chi if n is None else n)
    v[:len(k)] = np.exp(-12.0 * k / chi)
    return v / np.linalg.norm(v)


def _saturated_state(case, seed):
    """Every bond of rank chi with the same spectrum; across each odd bond the two
    Gammas are isometries over the outer Lambdas, as an update leaves them
    (Theta of that bond before the gate has exactly Lambda as its singular values)."""
    L, d, chi = case["L"], case["d"], case["chi"]
    g, dev = _generator(seed, 2)
    v = _spectrum(chi)
    w = torch.as_tensor(v, device=dev)
    gam = []
    for s in range(L):
        q, _ = torch.linalg.qr(_randn((d * chi, chi), g, dev))
        q = q.reshape(d, chi, chi) / w[None, :, None]  # (i, outer, inner)
        # site to the left of its odd bond: (a outer, i, b inner), else (a inner, i, b outer)
        gam.append(_pinned(q.permute(2, 0, 1) if s % 2 == 0 else q.permute(1, 0, 2)))
    return gam, [v.copy() for _ in range(L + 1)]


def _canonical_state(case, seed):
    """A normalised chain for the observables: every Gamma_s lambda_{s+1} a random
    isometry from the right, the last site closed on its first right index."""
    L, d, chi = case["L"], case["d"], case["chi"]
    g, dev = _generator(seed, 6)
    v = _spectrum(chi)
    w = torch.as_tensor(v, device=dev)
    gam = []
    for s in range(L):
        q, _ = torch.linalg.qr(_randn((d * chi, chi), g, dev))
        x = q.reshape(chi, d, chi) / w[:, None, None]  # (b, i, a)
        if s == L - 1:
            x[0] /= torch.linalg.vector_norm(x[0], dim=0)
        gam.append(_pinned(x))
    return gam, [v.copy() for _ in range(L + 1)]


def _nearby(case, seed, state):
    """The same state a little off, for the overlap."""
    g, dev = _generator(seed, 4)
    gam = [_pinned(torch.as_tensor(x.T, device=dev) * (1.0 + 0.01 * _randn(x.T.shape, g, dev))) for x in state[0]]
    return gam, state[1]


def _nc_counts(L, d, chi, N):
    """Kept Schmidt vectors per left particle number at every link: at most what
    the sites on either side can hold, spread around unit filling."""
    ways = [{0: 1}]
    for _ in range(L):
        nxt = {}
        for q, m in ways[-1].items():
            for n in range(d):
                nxt[q + n] = min(nxt.get(q + n, 0) + m, chi)
        ways.append(nxt)
    out = []
    for l in range(L + 1):
        cap = {q: min(ways[l].get(q, 0), ways[L - l].get(N - q, 0)) for q in range(N + 1)}
        cap = {q: m for q, m in cap.items() if m}
        w = {q: math.exp(-0.5 * ((q - l * N / L) / 1.3) ** 2) for q in cap}
        tot = sum(w.values())
        cnt = {q: min(cap[q], int(round(chi * w[q] / tot))) for q in cap}
        while sum(cnt.values()) > chi:
            cnt[max(cnt, key=cnt.get)] -= 1
        if not any(cnt.values()):
            cnt[min(cap, key=lambda q: abs(q - l * N / L))] = 1
        out.append({q: m for q, m in sorted(cnt.items()) if m})
    return out


def _nc_state(case, seed):
    """Block-sparse random Gammas over the particle numbers of _nc_counts (unit
    filling), every bond as full as its sites allow."""
    L, d, chi = case["L"], case["d"], case["chi"]
    N = L
    g, dev = _generator(seed, 3)
    rng = np.random.default_rng([seed, 3])
    ll, lr, lam = [], [], []
    for cnt in _nc_counts(L, d, chi, N):
        a = np.full(chi, 10000, dtype=np.int32)
        b = np.full(chi, 10000, dtype=np.int32)
        q = rng.permutation(np.concatenate([np.full(m, q) for q, m in cnt.items()]))
        a[:len(q)], b[:len(q)] = q, N - q
        ll.append(a)
        lr.append(b)
        lam.append(_spectrum(chi, len(q)))
    gam = []
    for s in range(L):
        qa, qb = torch.as_tensor(ll[s], device=dev), torch.as_tensor(ll[s + 1], device=dev)
        i = torch.arange(d, device=dev)
        ok = (qa[None, None, :] + i[None, :, None] == qb[:, None, None]) & (qb < 10000)[:, None, None]
        x = _randn((chi, d, chi), g, dev) * ok  # (b, i, a)
        w = torch.as_tensor(lam[s + 1], device=dev)
        n2 = (x.abs() ** 2 * (w ** 2)[:, None, None]).sum((0, 1))
        gam.append(_pinned(x / torch.sqrt(torch.where(n2 > 0, n2, torch.ones_like(n2)))[None, None, :]))
    return gam, lam, ll, lr


def _bond_state(case, seed):
    """Two sites between full bonds: the tensors of one update."""
    d, chi = case["d"], case["chi"]
    return _saturated_state({"L": 2, "d": d, "chi": chi}, seed)


def _bond_gate(case, seed):
    rng = np.random.default_rng([seed, 5])
    n = case["d"] ** 2
    h = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return _pkg().hamiltonians.matrix_exponential(0.5 * (h + h.conj().T), case["dt"])


def _state(case, seed):
    kind = case["kind"]
    if kind == "bond":
        return _bond_state(case, seed)
    if kind in ("quench", "ring"):
        return _product_state(case, seed)
    if kind == "nc":
        return _nc_state(case, seed)
    if kind == "measure":
        return _canonical_state(case, seed)
    return _saturated_state(case, seed)


# ---------------------------------------------------------------------------
# one case
# ---------------------------------------------------------------------------
def prepare(case, seed):
    pkg = _pkg()
    kind = case["kind"]
    L, d, chi = case.get("L", 2), case["d"], case["chi"]
    mode, form = FORMS[case.get("svd", "fp64")]
    if kind == "nc":
        chain = pkg.Chain(L, d, chi, mode=pkg.MODE_NC, tot_num=L, svd_mode=mode)
    else:
        chain = pkg.Chain(L, d, chi, svd_mode=mode)
    if form:
        chain.set_theta_form(form)
    st = {"case": dict(case), "chain": chain, "state": _state(case, seed)}
    if kind == "bond":
        st["gate"] = _bond_gate(case, seed)
    elif kind == "measure":
        st["H"] = _hamiltonian(case, seed)
        st["other"] = pkg.Chain(L, d, chi)
        st["other"].set_state(*_nearby(case, seed, st["state"]))
        chain.set_state(*st["state"])
    else:
        st["gates"] = _gates(case, seed)
    return st


def run(st):
    case, chain = st["case"], st["chain"]
    kind = case["kind"]
    if kind == "measure":  # the chain stays on the device
        return {"rho": chain.single_site_rho(), "energy": chain.local_energy(st["H"]),
                "entropy": chain.chain_entropy(), "overlap": np.array(chain.inner_product(st["other"]))}
    chain.set_state(*st["state"])
    if kind == "bond":
        te = chain.two_site_op(1, st["gate"])
        return {"kept": 1.0 - te, "lambda": chain.get_lambda(2), "rho2": chain.two_site_rho(1)}
    if kind == "sweep":
        links = list(range(1, case["L"], 2))
        kept = 1.0 - chain.apply_bonds(links, [st["gates"][l - 1] for l in links])
    elif kind == "ring":
        kept = np.array([1.0 - chain.trotter_step_pbc(st["gates"], case["order"]) for _ in range(case["steps"])])
    else:
        kept = np.array([1.0 - chain.trotter_step(st["gates"], case.get("order", 2))
                         for _ in range(case.get("steps", 1))])
    lam = np.zeros((case["L"] + 1, case["chi"]))
    for l in range(case["L"] + 1):
        chain.get_lambda_into(l + 1, lam[l])
    return {"kept": kept, "lambda": lam, "rho": chain.single_site_rho()}


def _updates(case):
    L = case.get("L", 2)
    odd, even = L // 2, (L - 1) // 2
    kind = case["kind"]
    if kind == "bond":
        return 1
    if kind == "sweep":
        return odd
    if kind == "nc":
        return 2 * odd + even
    if kind == "ring":
        return case["steps"] * (2 * odd + (2 if L % 2 else 1) * even + 2 * (L - 2) + 1)
    return case["steps"] * (2 * odd + even if case["order"] == 2 else 4 * odd + 3 * even)


def work(case):
    """Bytes: the chain in, the Gammas and Lambdas of every update read and written
    once, the results out.  Flops of an update: Theta, the gate, and the least a
    truncated SVD takes (a chi-wide factorisation of the Theta and its vectors).
    Ranks are those the state has; a quench's bonds are taken half full on
    average, a number-conserving Theta at the share of its allowed entries."""
    L, d, chi = case.get("L", 2), case["d"], case["chi"]
    gamma = 16.0 * d * chi * chi
    out = 8.0 * (L + 1) * chi + 16.0 * L * d * d
    if case["kind"] == "measure":
        theta = 8.0 * d * d * chi ** 3 + 8.0 * d ** 4 * chi ** 2
        return {"bytes": 2 * L * gamma + out, "flops": (L - 1) * theta + 16.0 * L * d * chi ** 3}
    r = chi / 2.0 if case["kind"] in ("quench", "ring") else float(chi)
    share = 1.0
    if case["kind"] == "nc":  # allowed (block) entries of a Theta whose numbers are spread over ~5 values
        share = 0.2
    n = d * r
    flops = share * (8.0 * n * n * r + 8.0 * d ** 4 * r * r + 3 * 8.0 * n * n * r)
    ups = _updates(case)
    return {"bytes": L * gamma + ups * 4 * 16.0 * d * r * r + out, "flops": ups * flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain numpy (LAPACK) and torch
# ---------------------------------------------------------------------------
_GUARD = float(np.float32(1e-15))


def _theta(l0, g1, l1, g2, l2):
    """(a, i, j, c) of lambda0 Gamma1 lambda1 Gamma2 lambda2"""
    chi, d, _ = g1.shape
    a = (l0[:, None, None] * g1 * l1).reshape(chi * d, chi)
    b = (g2 * l2).reshape(chi, d * chi)
    return (a @ b).reshape(chi, d, d, chi)


def _update(gam, lam, l, gate, normalise=True):
    """TwoSiteOp on sites l, l + 1 (0-based) of the lists, in place; the discarded weight."""
    g1, g2, l0, l2 = gam[l], gam[l + 1], lam[l], lam[l + 2]
    chi, d, _ = g1.shape
    th = _theta(l0, g1, lam[l + 1], g2, l2)
    th = np.einsum("pq,aqc->apc", gate, th.reshape(chi, d * d, chi)).reshape(chi, d, d, chi)
    if normalise:
        th = th / np.linalg.norm(th)
    u, s, vh = np.linalg.svd(th.reshape(chi * d, d * chi), full_matrices=False)
    s = s[:chi]
    keep = s > _GUARD
    norm = float(np.sum(s[keep] ** 2))
    lam[l + 1] = np.where(keep, s / math.sqrt(norm), 0.0)
    i0 = np.where(l0 > _GUARD, 1.0 / np.where(l0 > _GUARD, l0, 1.0), 0.0)
    i2 = np.where(l2 > _GUARD, 1.0 / np.where(l2 > _GUARD, l2, 1.0), 0.0)
    gam[l] = u[:, :chi].reshape(chi, d, chi) * i0[:, None, None]
    gam[l + 1] = vh[:chi].reshape(chi, d, chi) * i2
    return abs(1.0 - norm)


def _rho1(gam, lam):
    out = []
    for s, g in enumerate(gam):
        x = lam[s][:, None, None] * g * lam[s + 1]
        out.append(np.einsum("aib,ajb->ij", x, x.conj()))
    return np.array(out)


def exact(case, seed):
    kind = case["kind"]
    L, d, chi = case.get("L", 2), case["d"], case["chi"]
    if kind == "measure":
        return _exact_measure(case, seed)
    if kind in ("nc", "ring") or _updates(case) * (d * chi) ** 3 > 2e9:
        return None
    gam, lam = [list(x) for x in _state(case, seed)]
    if kind == "bond":
        te = _update(gam, lam, 0, _bond_gate(case, seed))
        th = _theta(lam[0], gam[0], lam[1], gam[1], lam[2]).reshape(chi, d * d, chi)
        return {"kept": 1.0 - te, "lambda": lam[1], "rho2": np.einsum("apc,aqc->pq", th, th.conj())}
    gates = _gates(case, seed)
    if kind == "sweep":
        kept = np.array([1.0 - _update(gam, lam, l, gates[l]) for l in range(0, L - 1, 2)])
    else:
        kept = []
        order = case.get("order", 2)
        pick = [1, 1, 2, 2, 2, 1, 1]
        for _ in range(case["steps"]):
            te = 0.0
            for s in range(3 if order == 2 else 7):
                for l in range(s % 2, L - 1, 2):
                    te += _update(gam, lam, l, gates[l if order == 2 else 2 * l + pick[s] - 1])
            kept.append(1.0 - te)
        kept = np.array(kept)
    return {"kept": kept, "lambda": np.array(lam), "rho": _rho1(gam, lam)}


def _exact_measure(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    L, d, chi = case["L"], case["d"], case["chi"]
    gam, lam = _canonical_state(case, seed)
    oth, olam = _nearby(case, seed, (gam, lam))
    H = _hamiltonian(case, seed)
    G = [torch.as_tensor(np.ascontiguousarray(g), device=dev) for g in gam]
    O = [torch.as_tensor(np.ascontiguousarray(g), device=dev) for g in oth]
    Lm = [torch.as_tensor(v, device=dev) for v in lam]
    Om = [torch.as_tensor(v, device=dev) for v in olam]
    energy = []
    for l in range(L - 1):
        a = (Lm[l][:, None, None] * G[l] * Lm[l + 1]).reshape(chi * d, chi)
        b = (G[l + 1] * Lm[l + 2]).reshape(chi, d * chi)
        th = (a @ b).reshape(chi, d * d, chi).permute(1, 0, 2).reshape(d * d, chi * chi)
        rho = th @ th.conj().T
        h = torch.as_tensor(np.asarray(H[l], dtype=np.complex128), device=dev)
        energy.append(float((h * rho.T).sum().real))
    E = torch.zeros((chi, chi), dtype=torch.complex128, device=dev)
    E[0, 0] = 1.0
    for s in range(L):
        x = (G[s] * Lm[s + 1]) if s < L - 1 else G[s]
        y = (O[s] * Om[s + 1]) if s < L - 1 else O[s]
        E = torch.einsum("xy,xia,yib->ab", E, x.conj(), y)
    entropy = np.array([-np.sum(v[v > 0] ** 2 * np.log(v[v > 0] ** 2)) / math.log(d) for v in lam])
    return {"rho": _rho1(gam, lam), "energy": np.array(energy), "entropy": entropy,
            "overlap": np.array(complex(E[0, 0].cpu()))}
