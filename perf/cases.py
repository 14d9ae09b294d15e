"""Performance cases of the two-electron engine: the calls a user's program makes, over the
range of sizes it makes them at, with an independent 64-bit evaluation of the small ones.

    listed()            the standing cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call: geometry, basis, context, density
    run(state)          one pass through the public entry points
    work(case)          bytes and flops the pass cannot do without
    exact(case, seed)   the same outputs in 64 bits from plain torch, for the cases small enough

Every input follows from the seed: the seed places the molecules and draws the densities.
"""
import math

import numpy as np
import torch

from chronusq_public_b200.aointegrals import (AOIntegrals, COULOMB, EXCHANGE, PREC_FP64, PREC_MIXED)
from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.batch import BatchAOIntegrals
from chronusq_public_b200.guess_model import NFEAT, PairMLP
from chronusq_public_b200.molecule import Molecule, single_water, water_cluster
from chronusq_public_b200.scf import SingleSlater, atomic_density

DEV = "cuda:0"


def listed():
    return [
        # The smallest use: one Fock build of one water, as every iteration of a small SCF
        # makes.  Latency and launches are all of it.
        {"name": "fock_water_631gd", "kind": "fock", "nwater": 1, "basis": "6-31g*"},
        # An open-shell diatomic: the UHF form, two densities in one pass over the integrals.
        {"name": "fock_o2_uhf_ccpvdz", "kind": "fock", "nwater": 0, "basis": "cc-pvdz", "uhf": True},
        # The drop-in call of a host program: numpy matrices through the list form (Coulomb and
        # exchange entries), copied in and out by the call.
        {"name": "contract_host_h2o5_631gd", "kind": "fock", "nwater": 5, "basis": "6-31g*", "host": True},
        # A medium cluster, an ordinary Fock build.
        {"name": "fock_h2o11_ccpvdz", "kind": "fock", "nwater": 11, "basis": "cc-pvdz"},
        # The benchmark's configuration: N = 768, every class up to (dd|dd).
        {"name": "fock_h2o32_ccpvdz", "kind": "fock", "nwater": 32, "basis": "cc-pvdz"},
        # One incremental build of the mixed-precision phase: a density change, FP32 quartets
        # below the cutoff, the looser screen of that phase.
        {"name": "fock_mixed_h2o20_ccpvdz", "kind": "fock", "nwater": 20, "basis": "cc-pvdz", "mixed": True},
        # Triple zeta: every class up to (ff|ff).
        {"name": "fock_h2o5_ccpvtz", "kind": "fock", "nwater": 5, "basis": "cc-pvtz"},
        # One iteration's Fock build of a batch of uneven clusters, as the batched SCF makes it:
        # the density copied in, one graph replay.
        {"name": "batch_40_631gd", "kind": "batch", "nmol": 40, "nmax": 12, "basis": "6-31g*"},
        # The one-electron set-up of an SCF in a static field: S, T, V and the dipole matrices.
        {"name": "one_e_h2o24_ccpvdz", "kind": "one_e", "nwater": 24, "basis": "cc-pvdz"},
        # A new geometry: basis upload and Schwarz bounds, once per molecule or geometry step.
        {"name": "setup_h2o10_ccpvdz", "kind": "setup", "nwater": 10, "basis": "cc-pvdz"},
        # A whole small SCF from the superposition of atomic densities to convergence.
        {"name": "scf_h2o2_631gd", "kind": "scf", "nwater": 2, "basis": "6-31g*"},
        # One step of the initial-guess network's training: forward, loss, backward, Adam.
        {"name": "guess_train_2048", "kind": "train", "batch": 2048, "maxf": 14},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    # Fock builds are most of what a user's program does, so half of the drawn cases are.
    kind = rng.choice(["fock"] * 6 + ["batch", "one_e", "setup", "scf", "train", "fock"])
    basis = rng.choice(["sto-3g", "6-31g", "6-31g*", "cc-pvdz", "cc-pvdz", "cc-pvtz"])
    if kind == "fock":
        nmax = {"cc-pvtz": 4, "cc-pvdz": 28}.get(basis, 30)
        c = {"kind": "fock", "nwater": _log_int(rng, 1, nmax), "basis": basis, "decay": round(rng.uniform(0.6, 1.2), 3)}
        form = rng.choice(["", "", "uhf", "host", "mixed"])
        if form:
            c[form] = True
        return c
    if kind == "batch":
        return {"kind": "batch", "nmol": _log_int(rng, 4, 40), "nmax": rng.randint(3, 12),
                "basis": rng.choice(["sto-3g", "6-31g", "6-31g*"])}
    if kind == "one_e":
        return {"kind": "one_e", "nwater": _log_int(rng, 1, 8 if basis == "cc-pvtz" else 24), "basis": basis}
    if kind == "setup":
        return {"kind": "setup", "nwater": _log_int(rng, 1, 4 if basis == "cc-pvtz" else 10), "basis": basis}
    if kind == "scf":
        return {"kind": "scf", "nwater": rng.randint(1, 2), "basis": rng.choice(["sto-3g", "6-31g", "6-31g*"])}
    return {"kind": "train", "batch": _log_int(rng, 200, 2048), "maxf": rng.choice([14, 30])}


# ------------------------------------------------------------------ inputs ---
def _molecule(case, seed):
    n = case["nwater"]
    if n == 0:   # O2, bond length around the experimental 1.21 Angstrom
        r = np.random.default_rng(seed).uniform(1.15, 1.27)
        return Molecule.from_angstrom([8, 8], [[0.0, 0.0, 0.0], [0.0, 0.0, r]], mult=3)
    return single_water(seed) if n == 1 else water_cluster(n, seed)


def _density(bs, rng, decay=0.8, scale=1.0):
    """Symmetric matrix with the fall-off of a molecular density: elements uniform in [-1, 1]
    times exp(-decay R), R the distance of the two functions' centres in bohr, and 1 more on
    the diagonal."""
    cent = np.concatenate([np.repeat(s.origin[None, :], s.size, axis=0) for s in bs.shells])
    R = np.linalg.norm(cent[:, None, :] - cent[None, :, :], axis=-1)
    u = rng.uniform(-1.0, 1.0, R.shape)
    D = 0.5 * (u + u.T) * np.exp(-decay * R)
    D[np.diag_indices_from(D)] += 1.0
    return np.ascontiguousarray(scale * D)


def _densities(case, bs, seed):
    rng = np.random.default_rng(seed)
    # an incremental build contracts the change between two iterations' densities
    scale = 1e-3 if case.get("mixed") else 1.0
    return [_density(bs, rng, case.get("decay", 0.8), scale) for _ in range(2 if case.get("uhf") else 1)]


def _batch_molecules(case, seed):
    # the sizes belong to the case, the geometries to the seed
    sizes = np.random.default_rng([case["nmol"], case["nmax"]]).integers(1, case["nmax"] + 1, size=case["nmol"])
    return [single_water(1000 * seed + i) if n == 1 else water_cluster(int(n), 1000 * seed + i)
            for i, n in enumerate(sizes)]


def _train_inputs(case, seed):
    rng = np.random.default_rng(seed)
    nout = case["maxf"] ** 2
    X = rng.standard_normal((case["batch"], NFEAT))
    T = rng.standard_normal((case["batch"], nout))
    # a pair's block fills the rows and columns its two atoms have (H: 5 of 14, 14 of 30)
    small = {14: 5, 30: 14}[case["maxf"]]
    na, nb = (np.where(rng.uniform(size=case["batch"]) < 0.4, case["maxf"], small) for _ in range(2))
    k = np.arange(case["maxf"])
    M = ((k[None, :, None] < na[:, None, None]) & (k[None, None, :] < nb[:, None, None])).reshape(-1, nout)
    return X, T, M.astype(np.float32)


def _weights(case, seed):
    """The network's starting weights, as its constructor draws them."""
    rng = np.random.default_rng(seed)
    dims = [NFEAT] + [256] * 4 + [case["maxf"] ** 2]
    W = [rng.normal(0.0, 1.0 / math.sqrt(dims[i]), size=(dims[i + 1], dims[i])) for i in range(5)]
    return W, [rng.normal(0.0, 0.01, size=d) for d in dims[1:]]


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "train":
        X, T, M = _train_inputs(case, seed)
        m = PairMLP(width=256, layers=4, seed=0, maxf=case["maxf"])
        m.set_weights(*_weights(case, seed))
        st.update(model=m, X=torch.tensor(X, dtype=torch.float32, device=DEV).to(torch.bfloat16),
                  T=torch.tensor(T, dtype=torch.float32, device=DEV), M=torch.tensor(M, device=DEV))
        return st
    if kind == "batch":
        bss = [BasisSet(case["basis"], m.atoms, m.coords) for m in _batch_molecules(case, seed)]
        B = BatchAOIntegrals(bss, thresholdSchwartz=1e-12)
        P = B.pack([_density(bs, np.random.default_rng([seed, i])) for i, bs in enumerate(bss)])
        # as the batched SCF: one build sizes the list, then the build is captured for replay
        B.formPT(P)
        B.enable_graph(int(1.25 * B.stats()["quartets"]) + 4096, 1)
        held, PT = P.clone(), B.zeros()
        st.update(B=B, P=P, held=held, PT=PT, graph=B.capture_formPT(held, PT, warm=False))
        return st
    mol = _molecule(case, seed)
    bs = BasisSet(case["basis"], mol.atoms, mol.coords)
    st.update(mol=mol, bs=bs)
    if kind == "scf":
        for z in set(mol.atoms):
            atomic_density(z, case["basis"], 0, 1e-12)   # kept by the program for every molecule
        st["hf"] = SingleSlater(mol, bs, thresholdSchwartz=1e-12)
        return st
    if kind == "setup":
        return st
    ints = AOIntegrals(bs)
    st["ints"] = ints
    if kind == "fock":
        Ds = _densities(case, bs, seed)
        if case.get("mixed"):
            ints.setPrecision(PREC_MIXED, 1e-8)
            ints.thresholdSchwartz = 1e-11
        else:
            ints.setPrecision(PREC_FP64)
        st["D"] = Ds if case.get("host") else [torch.tensor(D, device=DEV) for D in Ds]
    return st


# ------------------------------------------------------------------ one pass ---
def run(st):
    kind = st["kind"]
    if kind == "fock":
        ints, D = st["ints"], st["D"]
        if st["case"].get("host"):
            G = np.zeros_like(D[0])
            ints.newTwoEContractDirect([D[0], D[0]], [G, G], [COULOMB, EXCHANGE], [1.0, -0.5])
            return G
        return ints.formPT(D[0], D[1] if len(D) > 1 else None)
    if kind == "batch":
        st["held"].copy_(st["P"])
        st["graph"].replay()
        return st["PT"]
    if kind == "one_e":
        mol = st["mol"]
        S, T, V = st["ints"].computeAOOneE(mol.atoms, mol.coords, device_out=True)
        return S, T, V, st["ints"].computeDipole(device_out=True)
    if kind == "setup":
        ints = AOIntegrals(st["bs"])
        Q = ints.computeSchwartz()
        ints.close()
        return Q
    if kind == "scf":
        E = st["hf"].SCF3()
        return E, st["hf"].onePDMScalar
    m = st["model"]
    out, cache = m.forward(st["X"], keep=True)
    loss, dout = m.loss_grad(out, st["T"], st["M"], 1.0 / st["X"].shape[0])
    gW, gb = m.backward(dout, cache)
    m.adam(gW, gb, 2e-5)   # the learning rate of the first warm-up step
    return loss, gW, gb


# ------------------------------------------------------------------ necessary work ---
def work(case):
    """Bytes: each input matrix read and each output written once.  Flops: for the Fock
    builds the McMurchie-Davidson operation count of the quartets that pass the screen, as
    the engine's statistics report it; for the others the count given below."""
    kind = case["kind"]
    if kind == "train":
        nout, b = case["maxf"] ** 2, case["batch"]
        par = NFEAT * 256 + 3 * 256 * 256 + 256 * nout
        return {"bytes": 2.0 * b * NFEAT + 8.0 * b * nout + 36.0 * par, "flops": 6.0 * b * par}
    st = prepare(case, 1)
    try:
        if kind == "batch":
            B = st["B"]
            B.enable_graph(0)
            B.formPT(st["P"])
            return {"bytes": 16.0 * B.packed, "flops": B.stats()["model_flops"]}
        n = st["bs"].nbasis
        if kind == "fock":
            run(st)
            return {"bytes": 16.0 * n * n * len(st["D"]), "flops": st["ints"].stats()["model_flops"]}
        shells = st["bs"].shells
        if kind == "one_e":
            # per primitive pair and nucleus about 100 flops: Boys value, recursion, expansion
            nprim = sum(len(s.alpha) for s in shells)
            return {"bytes": 8.0 * 6 * n * n, "flops": 100.0 * nprim * (nprim + 1) / 2 * st["mol"].natoms}
        if kind == "setup":
            # about 100 flops for each pair of primitive pairs of a shell pair with itself
            k = np.array([len(s.alpha) for s in shells], dtype=float)
            return {"bytes": 8.0 * len(shells) ** 2, "flops": 50.0 * float((k ** 2).sum()) ** 2}
        hf = st["hf"]
        hf.SCF3()
        per = hf.ints.stats()["model_flops"] + 20.0 * n ** 3   # one build and the dense algebra
        return {"bytes": 16.0 * n * n, "flops": per * (hf.nSCFIter + 1)}
    finally:
        for k in ("ints", "B", "hf"):
            if k in st:
                st[k].close()


# ------------------------------------------------------------------ 64-bit evaluation ---
# McMurchie and Davidson, J. Comput. Phys. 26, 218 (1978), over all primitive pairs at once
# with torch; the basis set's exponents and normalised coefficients are inputs.
def _carts(l):
    return [(l - i, i - j, j) for i in range(l + 1) for j in range(i + 1)]


def _herms(n):
    return [c for t in range(n + 1) for c in _carts(t)]


def _harmonics(l):
    """Real solid harmonics m = -l..l over the Cartesians, each of the norm of x^l."""
    if l < 2:
        return np.eye(len(_carts(l)))
    s = math.sqrt
    rows = {2: [{(1, 1, 0): s(3)}, {(0, 1, 1): s(3)}, {(0, 0, 2): 1, (2, 0, 0): -.5, (0, 2, 0): -.5},
                {(1, 0, 1): s(3)}, {(2, 0, 0): s(3) / 2, (0, 2, 0): -s(3) / 2}],
            3: [{(2, 1, 0): 3 * s(5 / 8), (0, 3, 0): -s(5 / 8)}, {(1, 1, 1): s(15)},
                {(0, 1, 2): 4 * s(3 / 8), (2, 1, 0): -s(3 / 8), (0, 3, 0): -s(3 / 8)},
                {(0, 0, 3): 1, (2, 0, 1): -1.5, (0, 2, 1): -1.5},
                {(1, 0, 2): 4 * s(3 / 8), (3, 0, 0): -s(3 / 8), (1, 2, 0): -s(3 / 8)},
                {(2, 0, 1): s(15) / 2, (0, 2, 1): -s(15) / 2},
                {(3, 0, 0): s(5 / 8), (1, 2, 0): -3 * s(5 / 8)}]}[l]
    return np.array([[r.get(c, 0.0) for c in _carts(l)] for r in rows])


def _boys(nmax, T):
    """F_0..F_nmax: the ascending series for F_nmax and downward recursion below T = 35, the
    error function and upward recursion above."""
    lo = torch.clamp(T, max=35.0)
    term = torch.full_like(T, 1.0 / (2 * nmax + 1))
    tot = term.clone()
    for k in range(1, 130):
        term = term * (2.0 * lo / (2 * nmax + 2 * k + 1))
        tot = tot + term
    F = [None] * (nmax + 1)
    F[nmax] = torch.exp(-lo) * tot
    for n in range(nmax - 1, -1, -1):
        F[n] = (2.0 * lo * F[n + 1] + torch.exp(-lo)) / (2 * n + 1)
    hi = torch.clamp(T, min=35.0)
    U = 0.5 * torch.sqrt(math.pi / hi) * torch.erf(torch.sqrt(hi))
    for n in range(nmax + 1):
        F[n] = torch.where(T < 35.0, F[n], U)
        U = ((2 * n + 1) * U - torch.exp(-hi)) / (2.0 * hi)
    return F


def _hermite_coulomb(n, p, X):
    """R_tuv, t + u + v <= n, of exponent p and vector X (..., 3), in the order of _herms."""
    F = _boys(n, p * (X * X).sum(-1))
    lev = {(0, 0, 0): (-2.0 * p) ** n * F[n]}
    for m in range(n - 1, -1, -1):
        new = {(0, 0, 0): (-2.0 * p) ** m * F[m]}
        for c in _herms(n - m)[1:]:
            d = next(k for k in range(3) if c[k] > 0)
            a = tuple(c[k] - (k == d) for k in range(3))
            b = tuple(c[k] - 2 * (k == d) for k in range(3))
            new[c] = X[..., d] * lev[a] + ((c[d] - 1) * lev[b] if b[d] >= 0 else 0.0)
        lev = new
    return torch.stack([lev[c] for c in _herms(n)], -1)


class _PrimitivePairs:
    """The primitive pairs of all ordered shell pairs of one pair of angular momenta."""

    def __init__(self, bs, la, lb):
        prim = [(s, a, c, int(o)) for s, o in zip(bs.shells, bs.map_sh2bf) for a, c in zip(s.alpha, s.coef)]
        A, B = ([q for q in prim if q[0].l == l] for l in (la, lb))
        ia, ib = (x.reshape(-1) for x in np.meshgrid(np.arange(len(A)), np.arange(len(B)), indexing="ij"))

        def col(L, idx, f):
            v = np.array([f(q) for q in L], dtype=np.float64)
            return torch.tensor(v[idx], device=DEV)
        self.la, self.lb = la, lb
        self.a, self.b = col(A, ia, lambda q: q[1]), col(B, ib, lambda q: q[1])
        self.A, self.B = col(A, ia, lambda q: q[0].origin), col(B, ib, lambda q: q[0].origin)
        self.p = self.a + self.b
        self.P = (self.a[:, None] * self.A + self.b[:, None] * self.B) / self.p[:, None]
        AB2 = ((self.A - self.B) ** 2).sum(-1)
        self.K = (col(A, ia, lambda q: q[2]) * col(B, ib, lambda q: q[2]) * torch.exp(-self.a * self.b / self.p * AB2))
        oa, ob = np.array([q[3] for q in A])[ia], np.array([q[3] for q in B])[ib]
        na, nb = (len(_harmonics(l)) for l in (la, lb))
        self.fa = torch.tensor(oa[:, None] + np.repeat(np.arange(na), nb)[None], device=DEV)
        self.fb = torch.tensor(ob[:, None] + np.tile(np.arange(nb), na)[None], device=DEV)

    def expansion_1d(self, jmax):
        """E[d][i][j][t] for i <= la, j <= jmax."""
        h = 0.5 / self.p
        out = []
        for d in range(3):
            PA, PB = self.P[:, d] - self.A[:, d], self.P[:, d] - self.B[:, d]
            E = {(0, 0): [torch.ones_like(self.p)]}

            def step(prev, X):
                get = lambda t: prev[t] if 0 <= t < len(prev) else torch.zeros_like(self.p)   # noqa: E731
                return [X * get(t) + h * get(t - 1) + (t + 1) * get(t + 1) for t in range(len(prev) + 1)]
            for j in range(jmax + 1):
                if j > 0:
                    E[0, j] = step(E[0, j - 1], PB)
                for i in range(1, self.la + 1):
                    E[i, j] = step(E[i - 1, j], PA)
            out.append(E)
        return out

    def to_harmonics(self, M):
        """(pairs, cart_a cart_b, ...) to the basis functions."""
        ha, hb = (torch.tensor(_harmonics(l), device=DEV) for l in (self.la, self.lb))
        H = torch.kron(ha, hb)
        return torch.einsum("xc,nc...->nx...", H, M)

    def hermite(self):
        """Hermite expansion (pairs, functions, herms) of every product, coefficients included."""
        E = self.expansion_1d(self.lb)
        herm = _herms(self.la + self.lb)
        M = torch.zeros((len(self.p), len(_carts(self.la)) * len(_carts(self.lb)), len(herm)), dtype=torch.float64,
                        device=DEV)
        for x, (ca, cb) in enumerate((ca, cb) for ca in _carts(self.la) for cb in _carts(self.lb)):
            for k, tuv in enumerate(herm):
                if all(tuv[d] <= ca[d] + cb[d] for d in range(3)):
                    M[:, x, k] = self.K * math.prod(E[d][ca[d], cb[d]][tuv[d]] for d in range(3))
        return self.to_harmonics(M)


def _pair_groups(bs):
    ls = sorted({s.l for s in bs.shells})
    return [_PrimitivePairs(bs, a, b) for a in ls for b in ls]


def _exact_one_e(bs, Z, R):
    n = bs.nbasis
    Z, R = torch.tensor(np.array(Z, dtype=np.float64), device=DEV), torch.tensor(np.array(R), device=DEV)
    out = torch.zeros((6, n, n), dtype=torch.float64, device=DEV)
    for g in _pair_groups(bs):
        E = g.expansion_1d(g.lb + 2)
        s1 = torch.sqrt(math.pi / g.p)
        rows = []
        for ca in _carts(g.la):
            for cb in _carts(g.lb):
                S = [s1 * E[d][ca[d], cb[d]][0] for d in range(3)]
                T, D = [], []
                for d in range(3):
                    i, j = ca[d], cb[d]
                    t = -2.0 * g.b ** 2 * s1 * E[d][i, j + 2][0] + g.b * (2 * j + 1) * S[d]
                    T.append(t - 0.5 * j * (j - 1) * s1 * E[d][i, j - 2][0] if j > 1 else t)
                    e1 = E[d][i, j][1] if i + j > 0 else 0.0
                    D.append(s1 * e1 + g.P[:, d] * S[d])
                rows.append(torch.stack([
                    S[0] * S[1] * S[2], T[0] * S[1] * S[2] + S[0] * T[1] * S[2] + S[0] * S[1] * T[2],
                    D[0] * S[1] * S[2], S[0] * D[1] * S[2], S[0] * S[1] * D[2]], -1) * g.K[:, None])
        M = g.to_harmonics(torch.stack(rows, 1))
        for slot, k in ((0, 0), (1, 1), (3, 2), (4, 3), (5, 4)):
            out[slot].index_put_((g.fa, g.fb), M[..., k], accumulate=True)
        L = g.la + g.lb
        pot = torch.zeros((len(g.p), len(_herms(L))), dtype=torch.float64, device=DEV)
        for c in range(len(Z)):
            pot -= Z[c] * _hermite_coulomb(L, g.p, g.P - R[c])
        V = torch.einsum("nxh,nh->nx", g.hermite(), pot * (2.0 * math.pi / g.p)[:, None])
        out[2].index_put_((g.fa, g.fb), V, accumulate=True)
    return out[0], out[1], out[2], out[3:]


def _exact_eri(bs):
    """All (ab|cd) as an (n, n, n, n) tensor."""
    n = bs.nbasis
    eri = torch.zeros((n * n, n * n), dtype=torch.float64, device=DEV)
    groups = [(g, g.hermite()) for g in _pair_groups(bs)]
    for g, Eg in groups:
        hg = _herms(g.la + g.lb)
        for k, Ek in groups:
            hk = _herms(k.la + k.lb)
            pos = {c: i for i, c in enumerate(_herms(g.la + g.lb + k.la + k.lb))}
            idx = torch.tensor([[pos[tuple(x + y for x, y in zip(a, b))] for b in hk] for a in hg], device=DEV)
            sign = torch.tensor([(-1.0) ** sum(b) for b in hk], dtype=torch.float64, device=DEV)
            chunk = max(1, int(2e7 // (len(k.p) * idx.numel())))
            for s in range(0, len(g.p), chunk):
                p, q = g.p[s:s + chunk, None], k.p[None, :]
                X = g.P[s:s + chunk, None, :] - k.P[None, :, :]
                R = _hermite_coulomb(g.la + g.lb + k.la + k.lb, p * q / (p + q), X)
                R = R * (2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)))[..., None]
                W = torch.einsum("nmhk,myk->nhmy", R[:, :, idx] * sign, Ek)
                v = torch.einsum("nxh,nhmy->nxmy", Eg[s:s + chunk], W)
                half = torch.zeros((v.shape[0] * v.shape[1], n * n), dtype=torch.float64, device=DEV)
                half.index_add_(1, (k.fa * n + k.fb).reshape(-1), v.reshape(v.shape[0] * v.shape[1], -1))
                eri.index_add_(0, (g.fa * n + g.fb)[s:s + chunk].reshape(-1), half)
    return eri.view(n, n, n, n)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        X, T, M = _train_inputs(case, seed)
        W, b = ([torch.tensor(w, dtype=torch.float32, device=DEV) for w in v] for v in _weights(case, seed))
        W = [w.to(torch.bfloat16).double().requires_grad_() for w in W]
        b = [x.double().requires_grad_() for x in b]
        h = torch.tensor(X, dtype=torch.float32, device=DEV).to(torch.bfloat16).double()
        for i in range(len(W)):
            h = h @ W[i].T + b[i]
            h = torch.nn.functional.silu(h) if i + 1 < len(W) else h
        T, M = (torch.tensor(v, dtype=torch.float32, device=DEV).double() for v in (T, M))
        loss = (M * (h - T) ** 2).sum() / case["batch"]
        g = torch.autograd.grad(loss, W + b)
        return loss.detach().reshape(1), list(g[:5]), list(g[5:])
    if kind in ("batch", "scf"):
        return None
    mol = _molecule(case, seed)
    bs = BasisSet(case["basis"], mol.atoms, mol.coords)
    if kind == "one_e":
        return _exact_one_e(bs, mol.atoms, mol.coords)
    if bs.nbasis > 30:   # the integral tensor of the larger ones takes minutes
        return None
    I = _exact_eri(bs)
    if kind == "setup":
        Q = np.zeros((bs.nshell, bs.nshell))
        for i, a in enumerate(bs.shells):
            for j, c in enumerate(bs.shells):
                oa, oc = int(bs.map_sh2bf[i]), int(bs.map_sh2bf[j])
                blk = I[oa:oa + a.size, oc:oc + c.size, oa:oa + a.size, oc:oc + c.size]
                nn = a.size * c.size
                Q[i, j] = math.sqrt(float(blk.reshape(nn, nn).diagonal().abs().max()))
        return Q
    D = [torch.tensor(d, device=DEV) for d in _densities(case, bs, seed)]
    J = torch.einsum("abcd,cd->ab", I, D[0])
    K = [torch.einsum("acbd,cd->ab", I, d) for d in D]
    if case.get("host"):
        return 2.0 * J - K[0]
    return 2.0 * J - K[0], (-K[1] if len(D) > 1 else None)
