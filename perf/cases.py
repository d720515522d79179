"""The measured work of this library: builds, transforms and one-electron matrices through its
public entry points, over the sizes that its tests, its benchmark and its serving stream use.

A case is one call of an entry point for one molecular system (or one batch of systems):

  fock      LibintInterface_compute_2body_direct (host buffers) / LowdinGB300_twobody_device: the
            direct J/K matrix of an electron density, in FP64 or with the FP32/FP64 split
  batch     LowdinGB300_batch_fock: two-particle and coupling matrices of several systems
  coupling  LowdinGB300_coupling_device: both directions of the electron-proton Coulomb coupling
  quarter   LibintInterface_compute_2body_directIT: first-quarter transform of one orbital
  mp2       LowdinGB300_mp2_direct: closed-shell MP2 energy, FP64 or split-BF16 transform
  onebody   LowdinGB300_one_body_device: overlap, kinetic and point-charge matrices
  g12       libintinterface_compute_g12_direct: matrix of a Gaussian-geminal pair potential

Systems are the seeded generators of openlowdin_gb300.systems (water clusters, with or without a
d shell on O or quantum protons; H/C/N/O chains) and a generic contracted split-valence basis on
the same clusters.  The seed displaces the atoms slightly and mixes the occupied orbitals, so
other seeds are other molecules, other shell pairs and other densities of nearly the same cost.
"""
import math
import random

import numpy as np
import torch

from openlowdin_gb300 import flops as FL
from openlowdin_gb300 import lint as L
from openlowdin_gb300 import systems as S

EXACT_FUNCTIONS = 400        # exact(): largest basis of a dense table of integrals
GEMINAL = ([0.31, -0.12, 0.45], [0.6, 2.2, 7.5])   # coefficients, exponents


def listed():
    return [
        # one water molecule, the smallest SCF step through the reference-shaped host call: latency
        {"name": "fock-host-water1", "kind": "fock", "system": "water", "size": 1, "entry": "host",
         "precision": 0, "change": 1.0},
        # contracted split-valence basis with d on O, as ordinary inputs use: several primitives a shell
        {"name": "fock-host-contracted2", "kind": "fock", "system": "contracted", "size": 2, "entry": "host",
         "precision": 0, "change": 1.0},
        # four waters with a Cartesian d shell: classes up to (dd|dd)
        {"name": "fock-d-water4", "kind": "fock", "system": "water-d", "size": 4, "entry": "device",
         "precision": 0, "change": 1.0},
        # an ordinary s/p molecule of the serving stream, first build of a solve in FP64
        {"name": "fock-chain370", "kind": "fock", "system": "chain", "size": 370, "entry": "device",
         "precision": 0, "change": 1.0},
        # the upper part of the stream's sizes, FP32/FP64 split, a later iteration's density change
        {"name": "fock-mixed-chain700", "kind": "fock", "system": "chain", "size": 700, "entry": "device",
         "precision": 1, "change": 0.01},
        # eight four-water clusters with quantum protons, one batched build of an SCF iteration in FP64
        {"name": "batch-apmo8", "kind": "batch", "system": "apmo", "size": 4, "count": 8, "precision": 0},
        # electron-proton coupling of one cluster, all protons one species
        {"name": "coupling-water6", "kind": "coupling", "system": "apmo-single", "size": 6},
        # first quarter of the four-index transform for one orbital, host buffers (n^3 results)
        {"name": "quarter-water3", "kind": "quarter", "system": "water", "size": 3},
        # MP2 of a small cluster with d shells in FP64
        {"name": "mp2-d-water4", "kind": "mp2", "system": "water-d", "size": 4, "precision": 0},
        # MP2 of a large cluster on the split-BF16 tensor-core transform
        {"name": "mp2-split-d-water12", "kind": "mp2", "system": "water-d", "size": 12, "precision": 2},
        # one-electron matrices of a chain against all of its nuclei: once for each geometry
        {"name": "onebody-chain370", "kind": "onebody", "system": "chain", "size": 370},
        # geminal pair potential of the quantum-proton and fitted-potential inputs
        {"name": "g12-water2", "kind": "g12", "system": "water", "size": 2},
    ]


def draw(rng: random.Random):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fock", "fock", "fock", "mixed", "batch", "coupling", "quarter", "mp2", "mp2-split",
                       "onebody", "g12"])
    if kind in ("fock", "mixed"):
        precision = 1 if kind == "mixed" else 0
        system = rng.choice(["water", "water-d", "contracted", "chain", "chain"])
        entry = rng.choice(["host", "device"])
        size = (log_int(30, 700 if precision else 370) if system == "chain" else
                log_int(1, 8) if system == "water" else log_int(1, 4))
        return {"kind": "fock", "system": system, "size": size, "entry": entry, "precision": precision,
                "change": rng.choice([1.0, 0.1, 0.01, 0.001]) if precision else 1.0, "pick": rng.randrange(1000)}
    if kind == "batch":
        return {"kind": "batch", "system": rng.choice(["apmo", "chain", "water-d"]), "size": rng.randint(1, 3),
                "count": rng.randint(2, 8), "precision": rng.choice([0, 3]), "pick": rng.randrange(1000)}
    if kind == "coupling":
        return {"kind": "coupling", "system": "apmo-single", "size": rng.randint(1, 6), "pick": rng.randrange(1000)}
    if kind == "quarter":
        return {"kind": "quarter", "system": rng.choice(["water", "water-d", "contracted"]),
                "size": rng.randint(1, 3), "pick": rng.randrange(1000)}
    if kind == "mp2":
        return {"kind": "mp2", "system": rng.choice(["water", "water-d", "contracted"]), "size": rng.randint(1, 4),
                "precision": 0, "pick": rng.randrange(1000)}
    if kind == "mp2-split":
        return {"kind": "mp2", "system": rng.choice(["water", "water-d"]), "size": rng.randint(3, 10),
                "precision": rng.choice([1, 2]), "pick": rng.randrange(1000)}
    if kind == "onebody":
        system = rng.choice(["chain", "chain", "contracted"])
        return {"kind": "onebody", "system": system, "size": log_int(30, 370) if system == "chain" else log_int(1, 8),
                "pick": rng.randrange(1000)}
    return {"kind": "g12", "system": rng.choice(["water", "water-d"]), "size": rng.randint(1, 2),
            "pick": rng.randrange(1000)}


# ------------------------------------------------------------------ systems --
def _contracted_cluster(n, pick):
    """Water cluster in a generic contracted split-valence basis: O s 6/3/1, p 3/1, d 1; H s 3/1, p 1."""
    def contraction(lo, ratio, k):
        a = [lo * ratio ** (k - 1 - i) for i in range(k)]
        w = [math.exp(-0.35 * (i - 0.6 * k) ** 2) for i in range(k)]
        return a, w

    mols = S.cluster_positions(n, pick) if n > 1 else [S.water_geometry()]
    shells, Z, R = [], [], []
    for O, H1, H2 in mols:
        for l, lo, ratio, k in ((0, 5.0, 4.2, 6), (0, 0.9, 3.1, 3), (0, 0.27, 1.0, 1), (1, 0.8, 3.9, 3),
                                (1, 0.23, 1.0, 1), (2, 1.1, 1.0, 1)):
            a, w = contraction(lo, ratio, k)
            shells.append((l, a, w, list(O)))
        for H in (H1, H2):
            for l, lo, ratio, k in ((0, 0.6, 3.8, 3), (0, 0.16, 1.0, 1), (1, 1.1, 1.0, 1)):
                a, w = contraction(lo, ratio, k)
                shells.append((l, a, w, list(H)))
        Z += [8.0, 1.0, 1.0]
        R += [list(O), list(H1), list(H2)]
    return {"species": [S.electron_species(shells, 10 * n)], "point_charges": Z, "point_positions": R}


def _geometry(case, k=0):
    """The case's molecule number k before the seed's displacements."""
    pick, size, system = int(case.get("pick", 0)) + k, int(case["size"]), case["system"]
    if system == "chain":
        if case["kind"] == "batch":
            return S.chain_molecule(20_000 + pick, n_atoms=4 * size)
        return S.chain_for_basis(10_000 + pick, size) if size > 34 else S.chain_molecule(10_000 + pick, n_atoms=3)
    if system == "contracted":
        return _contracted_cluster(size, pick)
    if system in ("water", "water-d"):
        return S.water_cluster(size, seed=pick, o_d=system == "water-d", place=size > 1)
    mode = "single" if system == "apmo-single" else "per_proton"
    return S.water_cluster(size, seed=pick, quantum_protons=True, proton_species_mode=mode, place=size > 1)


def _molecule(case, seed, k=0):
    """Molecule k with every centre displaced by about 0.02 bohr, as the seed says."""
    m = _geometry(case, k)
    rng = np.random.default_rng([int(seed), k, 77])
    moved = {}

    def at(pos):
        key = tuple(round(float(x), 9) for x in pos)
        if key not in moved:
            moved[key] = [float(x) for x in np.asarray(pos, float) + rng.normal(scale=0.02, size=3)]
        return moved[key]

    m["point_positions"] = [at(p) for p in m["point_positions"]]
    for sp in m["species"]:
        sp["shells"] = [(l, a, c, at(o)) for l, a, c, o in sp["shells"]]
    return m


def _one_body(h, m):
    n = h.nbasis
    T = [torch.empty(n, n, dtype=torch.float64, device="cuda") for _ in range(3)]
    h.one_body_device(m["point_charges"], np.asarray(m["point_positions"]), *(t.data_ptr() for t in T),
                      stream=torch.cuda.current_stream().cuda_stream)
    return T


def _orbitals(h, sp, m, seed):
    """Orbital energies and coefficients (row p = orbital p) of a perturbed core Hamiltonian, and the
    number of occupied orbitals: what a first SCF iteration has in hand."""
    Sm, Tm, Vm = _one_body(h, m)
    torch.cuda.synchronize()
    q = float(sp["charge"])
    H = Tm / float(sp["mass"]) + q * Vm
    w, U = torch.linalg.eigh(Sm)
    keep = w > 1e-6 * w[-1]
    X = U[:, keep] / torch.sqrt(w[keep])
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    k = X.shape[1]
    N = torch.randn(k, k, dtype=torch.float64, device="cuda", generator=g)
    F = X.T @ H @ X + 0.02 * (N + N.T)
    e, V = torch.linalg.eigh(F)
    C = (X @ V).T.contiguous()
    if C.shape[0] < h.nbasis:   # near-dependent functions: pad with high virtual orbitals of zero coefficients
        C = torch.cat([C, torch.zeros(h.nbasis - k, h.nbasis, dtype=torch.float64, device="cuda")])
        e = torch.cat([e, e[-1] + 1.0 + torch.arange(h.nbasis - k, dtype=torch.float64, device="cuda")])
    nocc = max(1, int(round(sp["n_particles"] * sp["particles_fraction"])))
    return e, C, min(nocc, k - 1)


def _density(h, sp, m, seed):
    _, C, nocc = _orbitals(h, sp, m, seed)
    return sp["eta"] * (C[:nocc].T @ C[:nocc])


def prepare(case, seed):
    kind = case["kind"]
    st = torch.cuda.current_stream().cuda_stream
    if kind == "batch":
        mols = [_molecule(case, seed, k) for k in range(int(case["count"]))]
        handles = [[L.Libint2Interface(sp, i + 1) for i, sp in enumerate(m["species"])] for m in mols]
        total = sum(h.nbasis ** 2 for hs in handles for h in hs)
        P, G, J = (torch.zeros(total, dtype=torch.float64, device="cuda") for _ in range(3))
        b = L.Batch()
        at = 0
        for m, hs in zip(mols, handles):
            parts = [[], [], []]
            for i, (h, sp) in enumerate(zip(hs, m["species"])):
                n = h.nbasis
                for buf, part in zip((P, G, J), parts):
                    part.append(buf[at:at + n * n].view(n, n))
                parts[0][-1].copy_(_density(h, sp, m, seed + i))
                at += n * n
            b.add_system(hs, [sp["charge"] for sp in m["species"]],
                         [sp["kappa"] / sp["eta"] for sp in m["species"]],
                         [1 if sp["n_particles"] > 1 else 0 for sp in m["species"]], *parts)
        b.finalize(st)
        return {"case": case, "batch": b, "handles": handles, "P": P, "G": G, "J": J}
    m = _molecule(case, seed)
    sp = m["species"][0]
    h = L.Libint2Interface(sp, 1)
    n = h.nbasis
    state = {"case": case, "h": h, "m": m, "n": n}
    if kind == "onebody":
        state["out"] = [torch.empty(n, n, dtype=torch.float64, device="cuda") for _ in range(3)]
        state["Z"], state["R"] = np.array(m["point_charges"]), np.array(m["point_positions"])
        return state
    if kind == "coupling":
        p = m["species"][1]
        hp = L.Libint2Interface(p, 2)
        state.update(hp=hp, De=_density(h, sp, m, seed), Dp=_density(hp, p, m, seed + 1))
        state["Je"] = torch.empty(n, n, dtype=torch.float64, device="cuda")
        state["Jp"] = torch.empty(hp.nbasis, hp.nbasis, dtype=torch.float64, device="cuda")
        return state
    e, C, nocc = _orbitals(h, sp, m, seed)
    D = sp["eta"] * (C[:nocc].T @ C[:nocc])
    if kind == "fock":
        if case["change"] != 1.0:   # an incremental build takes the change of the density
            _, C2, _ = _orbitals(h, sp, m, seed + 1)
            D = case["change"] * (sp["eta"] * (C2[:nocc].T @ C2[:nocc]) - D)
        state["factor"] = sp["kappa"] / sp["eta"]
        if case["entry"] == "host":
            h.set_precision(case["precision"], 1e-5)
            state["D"] = D.cpu().numpy()
        else:
            state["D"] = D.contiguous()
            state["G"] = torch.empty(n, n, dtype=torch.float64, device="cuda")
    elif kind == "quarter":
        state.update(D=D.cpu().numpy(), C=C.cpu().numpy(), p=nocc - 1)
    elif kind == "mp2":
        state.update(D=D.contiguous(), C=C, e=e.cpu().numpy(), nocc=nocc, frozen=S.n_core(m))
    else:   # g12
        state.update(D=D.cpu().numpy(), factor=sp["kappa"] / sp["eta"])
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    st = torch.cuda.current_stream().cuda_stream
    if kind == "batch":
        state["batch"].fock(case["precision"], 1e-5 if case["precision"] else 0.0, st)
        return {"G": state["G"], "J": state["J"]}
    h = state["h"]
    if kind == "fock":
        if case["entry"] == "host":
            return h.compute_2body_direct(state["D"], state["factor"])
        h.twobody_device(state["D"].data_ptr(), state["G"].data_ptr(), state["factor"], case["precision"],
                         1e-5 if case["precision"] else 0.0, st)
        return state["G"]
    if kind == "coupling":
        L.coupling_device(h, state["hp"], state["De"].data_ptr(), state["Dp"].data_ptr(), state["Je"].data_ptr(),
                          state["Jp"].data_ptr(), stream=st)
        return {"Je": state["Je"], "Jp": state["Jp"]}
    if kind == "quarter":
        return h.compute_2body_directIT(state["D"], state["C"], state["p"])
    if kind == "mp2":
        return h.mp2_direct(state["D"].data_ptr(), state["C"].data_ptr(), state["e"], state["nocc"],
                            state["frozen"], case["precision"], stream=st)
    if kind == "onebody":
        h.one_body_device(state["Z"], state["R"], *(t.data_ptr() for t in state["out"]), stream=st)
        return state["out"]
    return h.compute_g12_direct(state["D"], state["factor"], *GEMINAL)


# --------------------------------------------------------------------- work --
def _pairs(shells, keep):
    """Significant shell pairs: {(la, lb): (estimated Schwarz factors, mean primitive pairs)}."""
    pos = np.array([s[3] for s in shells])
    low = np.array([min(s[1]) for s in shells])
    ls = np.array([s[0] for s in shells])
    npr = np.array([len(s[1]) for s in shells])
    i, j = np.tril_indices(len(shells))
    swap = ls[j] > ls[i]
    i, j = np.where(swap, j, i), np.where(swap, i, j)
    r2 = ((pos[i] - pos[j]) ** 2).sum(1)
    p = low[i] + low[j]
    q = (4 * low[i] * low[j] / p ** 2) ** 0.75 * np.exp(-low[i] * low[j] / p * r2) * p ** 0.25
    out = {}
    for la in range(4):
        for lb in range(la + 1):
            sel = (ls[i] == la) & (ls[j] == lb) & (q > keep)
            if sel.any():
                out[la, lb] = (q[sel], float((npr[i] * npr[j])[sel].mean()))
    return out


def _quartets(qa, qb, same, floor):
    """Pairs of pairs whose factors' product is over `floor`."""
    qb = np.sort(qb)
    n = float((len(qb) - np.searchsorted(qb, floor / qa)).sum())
    return n / 2 if same else n


def _integral_flops(bra, ket, kind, floor):
    """Recursion, transfer and digestion of every quartet over the floor (flops.quartet_flops)."""
    total = 0.0
    for (la, lb), (qa, na) in bra.items():
        for (lc, ld), (qb, nb) in ket.items():
            if bra is ket and (la, lb) < (lc, ld):
                continue
            n = _quartets(qa, qb, bra is ket and (la, lb) == (lc, ld), floor)
            total += n * FL.quartet_flops(la, lb, lc, ld, kind, na * nb)
    return total


def work(case):
    kind = case["kind"]
    if kind == "batch":
        got = {"bytes": 0.0, "flops": 0.0}
        for k in range(int(case["count"])):
            sp = _geometry(case, k)["species"]
            pairs = [_pairs(s["shells"], 1e-12) for s in sp]
            for a in range(len(sp)):
                got["bytes"] += 24.0 * S.nbasis(sp[a]) ** 2
                if sp[a]["n_particles"] > 1:
                    got["flops"] += _integral_flops(pairs[a], pairs[a], "jk", 2e-16)
                for b in range(a + 1, len(sp)):
                    got["flops"] += _integral_flops(pairs[a], pairs[b], "coupling", 1e-10)
        return got
    m = _geometry(case)
    sp = m["species"]
    n = float(S.nbasis(sp[0]))
    pairs = _pairs(sp[0]["shells"], 1e-12)
    if kind == "coupling":
        nb = float(S.nbasis(sp[1]))
        return {"bytes": 16 * (n * n + nb * nb),
                "flops": _integral_flops(pairs, _pairs(sp[1]["shells"], 1e-14), "coupling", 1e-10)}
    if kind == "fock":
        return {"bytes": 16 * n * n, "flops": _integral_flops(pairs, pairs, "jk", 2e-16 / max(case["change"], 1e-3))}
    if kind == "g12":
        return {"bytes": 16 * n * n, "flops": _integral_flops(pairs, pairs, "jk", 0.0)}
    if kind == "quarter":
        return {"bytes": 8 * (n ** 3 + n * n + n), "flops": _integral_flops(pairs, pairs, "jk", 1e-10)}
    if kind == "onebody":
        npair = sum(len(q) * k for q, k in pairs.values())
        return {"bytes": 24 * n * n, "flops": npair * (60.0 + 80.0 * len(m["point_charges"]))}
    o = max(1, sum(int(round(s["n_particles"] * s["particles_fraction"])) for s in sp) - S.n_core(m))
    v = n - o - S.n_core(m)
    cols = sum(len(q) * _ncart(a) * _ncart(b) for (a, b), (q, _) in pairs.items())
    gemms = 2.0 * (o * n * n * cols + o * v * n * cols + o * o * v * n * n + o * o * v * v * n)
    return {"bytes": 8 * (2 * n * n + n), "flops": 2 * _integral_flops(pairs, pairs, "none", 1e-10) + gemms}


def _ncart(l):
    return (l + 1) * (l + 2) // 2


# -------------------------------------------------------------------- exact --
# McMurchie-Davidson integrals over Hermite Gaussians in plain torch, FP64: every function pair is
# expanded in Hermite Gaussians about the product centres, the integral of two of them is R_tuv.
def _carts(l):
    return [(l - i, i - j, j) for i in range(l + 1) for j in range(i + 1)]


def _prim_norm(a, l):
    df = 1.0
    for k in range(2 * l - 1, 1, -2):
        df *= k
    return math.sqrt(2.0 ** l * (2 * a) ** (l + 1.5) / (math.pi ** 1.5 * df))


def _component_norms(shells):
    """1 / sqrt(self-overlap) of every function whose primitives carry the norm of x^l."""
    out = []
    for l, al, co, _ in shells:
        c = [w * _prim_norm(a, l) for a, w in zip(al, co)]
        for cart in _carts(l):
            s = 0.0
            for a, ca in zip(al, c):
                for b, cb in zip(al, c):
                    v = ca * cb * (math.pi / (a + b)) ** 1.5
                    for k in cart:
                        for f in range(2 * k - 1, 0, -2):
                            v *= f
                        v /= (2 * (a + b)) ** k
                    s += v
            out.append(1.0 / math.sqrt(s))
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _hermite_1d(i_max, j_max, PA, PB, p):
    """E[i, j][t] of one axis, without the Gaussian prefactor."""
    E = {(0, 0): [torch.ones_like(p)]}

    def up(e, x):
        n = len(e)
        get = lambda t: e[t] if 0 <= t < n else torch.zeros_like(p)  # noqa: E731
        return [get(t - 1) / (2 * p) + x * get(t) + (t + 1) * get(t + 1) for t in range(n + 1)]

    for i in range(i_max + 1):
        if i:
            E[i, 0] = up(E[i - 1, 0], PA)
        for j in range(1, j_max + 1):
            E[i, j] = up(E[i, j - 1], PB)
    return E


def _tuv(L_):
    return [(t, u, v) for s in range(L_ + 1) for t in range(s, -1, -1) for u in range(s - t, -1, -1)
            for v in (s - t - u,)]


class _PairTable:
    """Hermite expansions of all shell pairs, by class; column `base` of each pair's functions."""

    def __init__(self, shells):
        dev = dict(dtype=torch.float64, device="cuda")
        first, n = [], 0
        for l, *_ in shells:
            first.append(n)
            n += _ncart(l)
        self.n = n
        self.index = torch.zeros(n, n, dtype=torch.int64, device="cuda")
        groups, col = {}, 0
        index = np.zeros((n, n), dtype=np.int64)
        for i in range(len(shells)):
            for j in range(i + 1):
                a, b = (i, j) if shells[i][0] >= shells[j][0] else (j, i)
                na, nb = _ncart(shells[a][0]), _ncart(shells[b][0])
                block = col + np.arange(na * nb).reshape(na, nb)
                index[first[a]:first[a] + na, first[b]:first[b] + nb] = block
                if a != b:
                    index[first[b]:first[b] + nb, first[a]:first[a] + na] = block.T
                groups.setdefault((shells[a][0], shells[b][0]), []).append((a, b, col))
                col += na * nb
        self.ncol = col
        self.index = torch.tensor(index, device="cuda")
        self.classes = []
        for (la, lb), pairs in sorted(groups.items()):
            rows = [[], [], [], [], [], []]   # a, b, c, A, B, pair
            for k, (a, b, _) in enumerate(pairs):
                A, B = shells[a], shells[b]
                for x, cx in zip(A[1], A[2]):
                    for y, cy in zip(B[1], B[2]):
                        for r, v in zip(rows, (x, y, cx * _prim_norm(x, la) * cy * _prim_norm(y, lb), A[3], B[3], k)):
                            r.append(v)
            x, y, c, A, B = (torch.tensor(np.array(r), **dev) for r in rows[:5])
            p = x + y
            P = (x[:, None] * A + y[:, None] * B) / p[:, None]
            c = c * torch.exp(-x * y / p * ((A - B) ** 2).sum(1))
            E = [_hermite_1d(la, lb, P[:, d] - A[:, d], P[:, d] - B[:, d], p) for d in range(3)]
            herm = _tuv(la + lb)
            tab = torch.zeros(len(p), _ncart(la) * _ncart(lb), len(herm), **dev)
            for f, (ca, cb) in enumerate((u, v) for u in _carts(la) for v in _carts(lb)):
                ex = [E[d][ca[d], cb[d]] for d in range(3)]
                for h, tuv in enumerate(herm):
                    if all(tuv[d] < len(ex[d]) for d in range(3)):
                        tab[:, f, h] = c * ex[0][tuv[0]] * ex[1][tuv[1]] * ex[2][tuv[2]]
            base = torch.tensor([q[2] for q in pairs], device="cuda")
            self.classes.append({"L": la + lb, "p": p, "P": P, "E": tab, "herm": herm, "pairs": len(pairs),
                                 "pair": torch.tensor(rows[5], device="cuda"),
                                 "cols": base[:, None] + torch.arange(tab.shape[1], device="cuda")})


def _boys(m, T):
    """F_0..F_m(T), by the series of F_m and the downward recursion, or the upward one from erf."""
    small = T < 30.0
    Ts = torch.where(small, T, torch.ones_like(T))
    term = torch.full_like(T, 1.0 / (2 * m + 1))
    s = term.clone()
    for k in range(1, 140):
        term = term * (2 * Ts / (2 * m + 2 * k + 1))
        s = s + term
    e = torch.exp(-Ts)
    F = [None] * (m + 1)
    F[m] = e * s
    for k in range(m - 1, -1, -1):
        F[k] = (2 * Ts * F[k + 1] + e) / (2 * k + 1)
    Tl = torch.where(small, torch.full_like(T, 40.0), T)
    el = torch.exp(-Tl)
    U = 0.5 * torch.sqrt(math.pi / Tl) * torch.special.erf(torch.sqrt(Tl))
    for k in range(m + 1):
        F[k] = torch.where(small, F[k], U)
        U = ((2 * k + 1) * U - el) / (2 * Tl)
    return F


def _hermite_integrals(L_, start, X):
    """R_tuv (t + u + v <= L) from start[n] = R^(n)_000 and X = the three distances."""
    level = {(0, 0, 0): start}
    for t, u, v in _tuv(L_)[1:]:
        d = 0 if t else (1 if u else 2)
        low = [t, u, v]
        low[d] -= 1
        k = low[d]
        src = level[tuple(low)]
        low[d] -= 1
        lower = level[tuple(low)] if k else None
        level[t, u, v] = [X[d] * src[i + 1] + (k * lower[i + 1] if k else 0.0) for i in range(len(src) - 1)]
    return {key: val[0] for key, val in level.items()}


def _class_block(A, B, gem):
    """Contracted integrals of two pair classes: [pairs A, functions A, pairs B, functions B]."""
    Lt = A["L"] + B["L"]
    tuv = _tuv(Lt)
    where = {k: i for i, k in enumerate(tuv)}
    pick = torch.tensor([[where[tuple(x + y for x, y in zip(h, k))] for k in B["herm"]] for h in A["herm"]],
                        device="cuda")
    sign = torch.tensor([(-1.0) ** sum(k) for k in B["herm"]], dtype=torch.float64, device="cuda")
    nfa, nfb, nb = A["E"].shape[1], B["E"].shape[1], len(B["p"])
    out = torch.zeros(A["pairs"], nfa, B["pairs"], nfb, dtype=torch.float64, device="cuda")
    step = max(1, int(6e7 // (nb * max(pick.numel() + len(tuv) * 2, 200))))
    EB = B["E"] * sign
    for a0 in range(0, len(A["p"]), step):
        a = slice(a0, a0 + step)
        p, q = A["p"][a, None], B["p"][None, :]
        X = [A["P"][a, None, d] - B["P"][None, :, d] for d in range(3)]
        alpha = p * q / (p + q)
        T = alpha * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2)
        if gem is None:
            F = _boys(Lt, T)
        else:
            F = [torch.zeros_like(T) for _ in range(Lt + 1)]
            for c, g in zip(*gem):
                r = g / (alpha + g)
                v = 0.5 * math.sqrt(math.pi) * c * alpha * (alpha + g) ** -1.5 * torch.exp(-r * T)
                for k in range(Lt + 1):
                    F[k] = F[k] + v
                    v = v * r
        pref = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        R = _hermite_integrals(Lt, [pref * (-2 * alpha) ** k * f for k, f in enumerate(F)], X)
        R = torch.stack([R[k] for k in tuv])[pick]                  # [ha, hb, a, b]
        V = torch.einsum("afh,hkab,bgk->afbg", A["E"][a], R, EB)
        V = torch.zeros(V.shape[0], nfa, B["pairs"], nfb, dtype=V.dtype, device="cuda").index_add_(2, B["pair"], V)
        out.index_add_(0, A["pair"][a], V)
    return out


def _pair_matrix(ta, tb, gem=None):
    """Raw (ab|cd) over the function-pair columns of two tables."""
    M = torch.empty(ta.ncol, tb.ncol, dtype=torch.float64, device="cuda")
    for i, A in enumerate(ta.classes):
        for j, B in enumerate(tb.classes):
            if ta is tb and j > i:
                continue
            V = _class_block(A, B, gem).reshape(A["cols"].numel(), -1)
            ca, cb = A["cols"].reshape(-1), B["cols"].reshape(-1)
            M[ca[:, None], cb[None, :]] = V
            if ta is tb and j < i:
                M[cb[:, None], ca[None, :]] = V.T
    return M


def _two_body(M, t, N, D, f):
    """J + f K of the raw pair integrals M and the density D, N the component norms."""
    Ds = (D * N[:, None] * N[None, :]).contiguous()
    n = t.n
    J = torch.empty(n, n, dtype=torch.float64, device="cuda")
    K = torch.empty_like(J)
    for a in range(n):
        V = M[t.index[a]][:, t.index]       # [b, c, d] = (ab|cd)
        J[a] = (V.reshape(n, -1) @ Ds.reshape(-1, 1))[:, 0]
        K[a] = torch.einsum("rqs,rs->q", V, Ds)
    return (J + f * K) * N[:, None] * N[None, :]


def _exact_onebody(m):
    sp = m["species"][0]
    t = _PairTable(sp["shells"])
    N = _component_norms(sp["shells"])
    R = torch.tensor(m["point_positions"], dtype=torch.float64, device="cuda")
    raised = [[], []]
    Sv = torch.zeros(t.ncol, dtype=torch.float64, device="cuda")
    Vv = torch.zeros_like(Sv)
    for A in t.classes:
        s = A["E"][:, :, 0] * (math.pi / A["p"])[:, None] ** 1.5
        Sv.index_add_(0, A["cols"][A["pair"]].reshape(-1), s.reshape(-1))
        for z, C in zip(m["point_charges"], R):
            X = [A["P"][:, d] - C[d] for d in range(3)]
            F = _boys(A["L"], A["p"] * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2))
            H = _hermite_integrals(A["L"], [2 * math.pi / A["p"] * z * (-2 * A["p"]) ** k * f
                                            for k, f in enumerate(F)], X)
            H = torch.stack([H[k] for k in A["herm"]], 1)
            Vv.index_add_(0, A["cols"][A["pair"]].reshape(-1), torch.einsum("pfh,ph->pf", A["E"], H).reshape(-1))
    # kinetic energy: -1/2 d2/dx2 of x^j exp(-b x^2) is a sum of overlaps with j - 2, j and j + 2
    shells = sp["shells"]
    first, n = [], 0
    for l, *_ in shells:
        first.append(n)
        n += _ncart(l)
    T = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    groups = {}
    for i, A in enumerate(shells):
        for j, B in enumerate(shells):
            for x, cx in zip(A[1], A[2]):
                for y, cy in zip(B[1], B[2]):
                    groups.setdefault((A[0], B[0]), []).append(
                        (x, y, cx * _prim_norm(x, A[0]) * cy * _prim_norm(y, B[0]), *A[3], *B[3], first[i], first[j]))
    for (la, lb), rows in groups.items():
        d = torch.tensor(np.array([r[:9] for r in rows]), dtype=torch.float64, device="cuda")
        fi, fj = (torch.tensor([r[k] for r in rows], device="cuda") for k in (9, 10))
        x, y, c, A, B = d[:, 0], d[:, 1], d[:, 2], d[:, 3:6], d[:, 6:9]
        p = x + y
        P = (x[:, None] * A + y[:, None] * B) / p[:, None]
        c = c * torch.exp(-x * y / p * ((A - B) ** 2).sum(1)) * (math.pi / p) ** 1.5
        E = [_hermite_1d(la, lb + 2, P[:, k] - A[:, k], P[:, k] - B[:, k], p) for k in range(3)]
        s1 = lambda k, i, j: E[k][i, j][0]  # noqa: E731

        def t1(k, i, j):
            v = y * (2 * j + 1) * s1(k, i, j) - 2 * y * y * s1(k, i, j + 2)
            return v - 0.5 * j * (j - 1) * s1(k, i, j - 2) if j > 1 else v

        for u, ca in enumerate(_carts(la)):
            for w, cb in enumerate(_carts(lb)):
                o = [s1(k, ca[k], cb[k]) for k in range(3)]
                v = sum(t1(k, ca[k], cb[k]) * o[(k + 1) % 3] * o[(k + 2) % 3] for k in range(3))
                T.view(-1).index_add_(0, (fi + u) * n + fj + w, c * v)
    nn = N[:, None] * N[None, :]
    return [Sv[t.index] * nn, T * nn, Vv[t.index] * nn]


def _coupling_matrices(a, b, Da, Db):
    """J of species a from Db and of species b from Da; a, b: (pair table, component norms).  The
    library's integral set: raw values below 1e-10 are dropped."""
    M = _pair_matrix(a[0], b[0])
    M[M.abs() < 1e-10] = 0.0

    def j(M, ta, Na, tb, Nb, D):
        w = torch.zeros(tb.ncol, dtype=torch.float64, device="cuda")
        w.index_add_(0, tb.index.reshape(-1), (D * Nb[:, None] * Nb[None, :]).reshape(-1))
        return (M @ w[:, None])[:, 0][ta.index] * Na[:, None] * Na[None, :]

    return j(M, *a, *b, Db), j(M.T.contiguous(), *b, *a, Da)


def _exact_batch(case, seed):
    state = prepare(case, seed)
    G, J = torch.zeros_like(state["G"]), torch.zeros_like(state["J"])
    at = 0
    for k, hs in enumerate(state["handles"]):
        sp = _molecule(case, seed, k)["species"]
        tabs = [(_PairTable(s["shells"]), _component_norms(s["shells"])) for s in sp]
        view = []
        for h in hs:
            view.append([buf[at:at + h.nbasis ** 2].view(h.nbasis, h.nbasis) for buf in (state["P"], G, J)])
            at += h.nbasis ** 2
        for i, a in enumerate(sp):
            if a["n_particles"] > 1:
                M = _pair_matrix(tabs[i][0], tabs[i][0])
                view[i][1].copy_(a["charge"] ** 2 * _two_body(M, *tabs[i], view[i][0], a["kappa"] / a["eta"]))
            for j in range(i + 1, len(sp)):
                Ji, Jj = _coupling_matrices(tabs[i], tabs[j], view[i][0], view[j][0])
                q = a["charge"] * sp[j]["charge"]
                view[i][2].add_(q * Ji)
                view[j][2].add_(q * Jj)
    return {"G": G, "J": J}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    m = _molecule(case, seed)
    sp = m["species"][0]
    if kind == "onebody":
        return _exact_onebody(m)
    if S.nbasis(sp) > (EXACT_FUNCTIONS if kind == "fock" else 210):
        return None
    state = prepare(case, seed)
    t = _PairTable(sp["shells"])
    N = _component_norms(sp["shells"])
    if kind == "coupling":
        p = m["species"][1]
        Je, Jp = _coupling_matrices((t, N), (_PairTable(p["shells"]), _component_norms(p["shells"])), state["De"],
                                    state["Dp"])
        return {"Je": Je, "Jp": Jp}
    M = _pair_matrix(t, t, GEMINAL if kind == "g12" else None)
    dev = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    if kind in ("fock", "g12"):
        G = _two_body(M, t, N, dev(state["D"]), state["factor"])
        return G if case.get("entry") == "device" else G.cpu().numpy()
    M[M.abs() <= 1e-10] = 0.0    # the transforms' integral set
    n = t.n
    if kind == "quarter":
        Cs = dev(state["C"])[state["p"]] * N
        out = torch.stack([torch.einsum("m,mls->ls", Cs, M[t.index[:, nu]][:, t.index]) for nu in range(n)])
        return (out * N[:, None, None] * N[None, :, None] * N[None, None, :]).cpu().numpy()
    C = state["C"] * N
    e = dev(state["e"])
    o, v = C[state["frozen"]:state["nocc"]], C[state["nocc"]:]
    eo, ev = e[state["frozen"]:state["nocc"]], e[state["nocc"]:]
    half = torch.empty(len(o) * len(v), t.ncol, dtype=torch.float64, device="cuda")
    for k in range(0, t.ncol, 2000):
        A = M[:, k:k + 2000][t.index]                        # [mu, nu, column]
        A = torch.einsum("im,mnc->inc", o, A)
        half[:, k:k + 2000] = torch.einsum("an,inc->iac", v, A).reshape(len(half), -1)
    full = torch.empty(len(half), len(o), len(v), dtype=torch.float64, device="cuda")
    for k in range(0, len(half), 256):
        B = half[k:k + 256][:, t.index]                      # [ia, lam, sig]
        full[k:k + 256] = torch.einsum("jl,xls,bs->xjb", o, B, v)
    I = full.reshape(len(o), len(v), len(o), len(v))
    I[I.abs() <= 1e-10] = 0.0
    gap = eo[:, None, None, None] + eo[None, None, :, None] - ev[None, :, None, None] - ev[None, None, None, :]
    return float((I * (2 * I - I.permute(0, 3, 2, 1)) / gap).sum())
