"""The work that users of this framework have it do, as timed cases.

Each case is one pass through a public entry point, on inputs of the sizes
that the repository's own workloads have (water clusters and alkanes in
STO-3G / 6-31G* / 6-31G**, water to C16H34) and on everything between:

    fock      get2JmK on integral-direct Ints, the reference's own call
              (numpy density in, numpy G out), or DirectInts.jk on the GPU
    coulomb   DirectInts.j: the J of a DFT iteration
    uhf       getJK2: both spin densities of a UHF iteration
    ints      get2ints: every unique (ij|kl) packed, for a stored-integral SCF
    stored    get2JmK on stored packed integrals
    gradient  the analytic RHF gradient of a converged density
    mp2       the MP2 energy from packed integrals
    xc        one DFT iteration's grid work: density, functional, Fxc
    oneint    get1ints: S and h = T + V
    batch     batched_rhf: whole SCFs of a set of molecules

``exact`` restates the integrals by McMurchie--Davidson expansions in plain
64-bit torch (differentiable, so the gradient is its autograd), which is
affordable for the small molecules; the packed arrays of ``stored`` and
``mp2`` are three-index products, whose J, K and MO integrals have a
closed form at every size.
"""
import itertools
import math

import numpy as np
import torch

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # a small molecule, where an SCF step is all latency
        dict(name="fock_water_host", kind="fock", mol="water", n=1, basis="6-31g**", precision="fp64", host=True),
        # the headline workload: one Fock build of an RHF on (H2O)8, PyQuante's call
        dict(name="fock_h2o8_host", kind="fock", mol="water", n=8, basis="6-31g**", precision="fp64", host=True),
        # the largest molecule, mixed precision, density and result kept on the GPU
        dict(name="fock_c16h34_mixed", kind="fock", mol="alkane", n=16, basis="6-31g*", precision="mixed", host=False),
        # the Coulomb build of a DFT iteration (no exchange)
        dict(name="coulomb_c8h18", kind="coulomb", mol="alkane", n=8, basis="6-31g**", precision="fp64"),
        # a UHF iteration's J and K of two densities
        dict(name="uhf_h2o5", kind="uhf", mol="water", n=5, basis="6-31g*", precision="fp64"),
        # all packed integrals of a stored-integral SCF or an MP2
        dict(name="ints_h2o6", kind="ints", mol="water", n=6, basis="6-31g**"),
        # an iteration of a stored-integral SCF at (H2O)8's size
        dict(name="stored_fock_200", kind="stored", nbf=200),
        # the gradient of a geometry optimisation's step
        dict(name="gradient_h2o4", kind="gradient", mol="water", n=4, basis="6-31g*", precision="fp64"),
        # an MP2 energy at (H2O)6's size
        dict(name="mp2_150", kind="mp2", nbf=150, nocc=30),
        # a DFT iteration's functional and Fxc on the default grid
        dict(name="xc_h2o8", kind="xc", mol="water", n=8, basis="6-31g**"),
        # overlap and core Hamiltonian, once per geometry of every calculation
        dict(name="oneint_c16h34", kind="oneint", mol="alkane", n=16, basis="6-31g*"),
        # many small molecules solved together
        dict(name="batch_32", kind="batch", count=32, kmax=5),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))))


def draw(rng):
    given = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        c = _drawn(rng)
        if c not in given:
            return c


def _drawn(rng):
    kind = rng.choice(["fock", "fock", "coulomb", "uhf", "ints", "stored", "gradient", "mp2", "xc", "oneint", "batch"])
    c = dict(kind=kind)
    if kind == "stored":
        c.update(nbf=_log_int(rng, 7, 200))
    elif kind == "mp2":
        c.update(nbf=_log_int(rng, 13, 150))
        c.update(nocc=max(1, int(c["nbf"] * rng.uniform(0.15, 0.4))))
    elif kind == "batch":
        c.update(count=_log_int(rng, 3, 32), kmax=rng.randint(1, 5))
    else:
        top = dict(fock=(8, 16), coulomb=(6, 8), uhf=(5, 6), ints=(6, 6), gradient=(4, 5), xc=(8, 8), oneint=(8, 16))[kind]
        c.update(mol=rng.choice(["water", "alkane"]))
        c.update(n=_log_int(rng, 1 if c["mol"] == "water" else 2, top[c["mol"] == "alkane"]))
        # (the largest sizes above are for 6-31G*: 6-31G** only below them)
        bases = ["sto-3g", "6-31g*"] + (["6-31g**"] if c["mol"] == "water" or c["n"] < top[1] - 2 else [])
        c.update(basis=rng.choice(bases))
        if kind in ("fock", "coulomb", "uhf", "gradient"):
            c.update(precision=rng.choice(["fp64", "mixed"]))
        if kind == "fock":
            c.update(host=rng.random() < 0.5)
    return c


# ---------------------------------------------------------------- inputs --

def _molecule(case, seed):
    from pyquante_b200 import geometries
    if case["mol"] == "water":
        return geometries.water_cluster(case["n"], seed=seed)
    return geometries.perturbed(geometries.alkane(case["n"]), 0.05, seed)


def _basis(case, seed):
    from pyquante_b200.Basis.basis import BasisSet
    mol = _molecule(case, seed)
    return mol, BasisSet(mol, case["basis"])


def _guess(mol, bs, nocc=None):
    """Occupied orbitals (n x nocc) and energies of the core Hamiltonian."""
    ref = _Reference(mol, bs)
    S, T, V = ref.one_electron(ref.R)
    L = torch.linalg.cholesky(S)
    Li = torch.linalg.inv(L)
    e, U = torch.linalg.eigh(Li @ (T + V) @ Li.T)
    nocc = mol.get_nel() // 2 if nocc is None else nocc
    return (Li.T @ U)[:, :nocc].contiguous(), e[:nocc].contiguous()


def _three_index(nbf, seed):
    """b[Q, pair(i, j)] with (ij|kl) = sum_Q b[Q, ij] b[Q, kl]: functions at
    seeded places, overlaps falling off with their distance, as integrals over
    Gaussians do."""
    g = torch.Generator().manual_seed(int(seed))
    naux = 2 * nbf
    box = 2.0 * nbf ** (1.0 / 3.0)
    x = (torch.rand(nbf, 3, generator=g, dtype=F64) * box).to(DEV)
    y = (torch.rand(naux, 3, generator=g, dtype=F64) * box).to(DEV)
    noise = torch.randn(naux, nbf * (nbf + 1) // 2, generator=g, dtype=torch.float32).to(DEV).to(F64)
    i, j = torch.tril_indices(nbf, nbf, device=DEV)
    d2 = (x[i] - x[j]).square().sum(1)
    mid = 0.5 * (x[i] + x[j])
    return noise * torch.exp(-0.25 * d2)[None, :] / (1.0 + torch.cdist(y, mid).square())


def _pack(b):
    """The packed array of sum_Q b[Q, IJ] b[Q, KL], KL <= IJ."""
    P = b.shape[1]
    out = torch.empty(P * (P + 1) // 2, dtype=F64, device=DEV)
    for r0 in range(0, P, 2048):
        r1 = min(P, r0 + 2048)
        m = b[:, r0:r1].T @ b[:, :r1]
        keep = torch.arange(r1, device=DEV)[None, :] <= torch.arange(r0, r1, device=DEV)[:, None]
        out[r0 * (r0 + 1) // 2:r1 * (r1 + 1) // 2] = m[keep]
    return out


def _orbitals(nbf, nocc, seed):
    g = torch.Generator().manual_seed(int(seed) + 7)
    C = torch.linalg.qr(torch.randn(nbf, nbf, generator=g, dtype=F64))[0]
    eo = torch.sort(-0.4 - 1.2 * torch.rand(nocc, generator=g, dtype=F64))[0]
    ev = torch.sort(0.15 + 3.0 * torch.rand(nbf - nocc, generator=g, dtype=F64))[0]
    return C.contiguous().to(DEV), torch.cat([eo, ev]).to(DEV)


def _stored_density(nbf, seed):
    C, _ = _orbitals(nbf, max(1, nbf // 5), seed)
    Co = C[:, :max(1, nbf // 5)]
    return (Co @ Co.T).contiguous()


def _systems(case, seed):
    from pyquante_b200 import geometries
    return geometries.cluster_batch(case["count"], seed=seed, kmax=case["kmax"])


def prepare(case, seed):
    from pyquante_b200 import Ints
    k = case["kind"]
    s = dict(kind=k, case=case)
    if k == "stored":
        s.update(ints=_pack(_three_index(case["nbf"], seed)), D=_stored_density(case["nbf"], seed))
    elif k == "mp2":
        C, e = _orbitals(case["nbf"], case["nocc"], seed)
        s.update(ints=_pack(_three_index(case["nbf"], seed)), orbs=C.cpu().numpy(), orbe=e.cpu().numpy())
    elif k == "batch":
        s.update(systems=_systems(case, seed))
    else:
        mol, bs = _basis(case, seed)
        s.update(mol=mol, bfs=bs)
        if k in ("fock", "coulomb", "uhf"):
            s.update(ints=Ints.get2ints(bs, direct=True, precision=case["precision"]))
            C, _ = _guess(mol, bs)
            D = (C @ C.T).contiguous()
            if k == "uhf":
                Cb = C[:, :max(1, C.shape[1] - 1)]
                s.update(Da=D, Db=(Cb @ Cb.T).contiguous())
            else:
                s.update(D=D.cpu().numpy() if case.get("host") else D)
        elif k == "gradient":
            s.update(ints=Ints.get2ints(bs, direct=True, precision=case["precision"]))
            C, e = _guess(mol, bs)
            s.update(D=(C @ C.T).contiguous(), W=((C * e) @ C.T).contiguous())
        elif k == "xc":
            from pyquante_b200.MolecularGrid import MolecularGrid
            s.update(grid=MolecularGrid(mol))
            s["grid"].set_bf_amps(bs)
            C, _ = _guess(mol, bs)
            s.update(D=(C @ C.T).contiguous())
    return s


def run(s):
    from pyquante_b200 import Ints
    k, case = s["kind"], s["case"]
    if k == "fock":
        return Ints.get2JmK(s["ints"], s["D"]) if case["host"] else s["ints"].jk(s["D"])
    if k == "coulomb":
        return s["ints"].j(s["D"])
    if k == "uhf":
        return Ints.getJK2(s["ints"], s["Da"], s["Db"])
    if k == "ints":
        return Ints.get2ints(s["bfs"]).tensor
    if k == "stored":
        return Ints.get2JmK(s["ints"], s["D"])
    if k == "gradient":
        from pyquante_b200.force import rhf_gradient_from_density
        return rhf_gradient_from_density(s["mol"], s["ints"].engine, s["D"], s["W"], case["precision"])
    if k == "mp2":
        from pyquante_b200.MP import MP2
        return MP2(s["ints"], s["orbs"], s["orbe"], case["nocc"], case["nbf"] - case["nocc"])
    if k == "xc":
        from pyquante_b200.dft import getXC
        s["grid"].setdens(s["D"])
        exc, fxc = getXC(s["grid"], s["mol"].get_nel())
        return dict(exc=exc, fxc=fxc, density=s["grid"].density)
    if k == "oneint":
        return Ints.get1ints(s["bfs"], s["mol"].atoms)
    if k == "batch":
        from pyquante_b200.batch import batched_rhf
        return batched_rhf(s["systems"])["energies"]
    raise ValueError(k)


# ------------------------------------------------------------------ work --

def _plan_flops(eng):
    """FP64 operations of the primitive quartets that a screened build keeps."""
    import ctypes
    from pyquante_b200 import flops
    q, p = (ctypes.c_int64 * 42)(), (ctypes.c_int64 * 42)()
    eng.ctx.check(eng.ctx.lib.pqb_plan_stats(eng.ctx.h, q, p))
    return float(sum(p[x] * flops.prim_quartet_flops(*flops.quartet_class_ls(x % 21)) for x in range(42)))


def _all_flops(bs):
    """The same for every unique shell quartet, unscreened."""
    from pyquante_b200 import flops
    sh = [(sum(s.functions[0].powers), len(s.functions[0].pexps)) for s in bs.shells]
    per = {}
    for a in range(len(sh)):
        for b in range(a + 1):
            key = tuple(sorted((sh[a][0], sh[b][0]), reverse=True))
            n, n2 = per.get(key, (0, 0))
            k = sh[a][1] * sh[b][1]
            per[key] = (n + k, n2 + k * k)
    total = 0.0
    for x, y in itertools.combinations_with_replacement(sorted(per, reverse=True), 2):
        count = (per[x][0] ** 2 + per[x][1]) / 2 if x == y else per[x][0] * per[y][0]
        total += count * flops.prim_quartet_flops(*x, *y)
    return total


def work(case):
    k = case["kind"]
    if k in ("stored", "mp2"):
        n = case["nbf"]
        P = n * (n + 1) // 2
        Q = P * (P + 1) // 2
        if k == "stored":
            return dict(bytes=8.0 * (Q + 2 * n * n), flops=12.0 * Q)
        o, v = case["nocc"], n - case["nocc"]
        return dict(bytes=8.0 * (Q + n * n), flops=2.0 * (P * n * o * (n + v) + o * o * v * n * n / 2 + o * o * v * v * n / 2))
    from pyquante_b200 import Ints
    if k == "batch":
        from pyquante_b200.batch import BatchEngine
        eng = BatchEngine(_systems(case, 1))
        eng.plan()
        return dict(bytes=8.0 * 3 * eng.dense_len, flops=12.0 * _plan_flops(eng))   # about twelve iterations
    mol, bs = _basis(case, 1)
    n, nat = len(bs), len(mol.atoms)
    if k == "ints":
        P = n * (n + 1) // 2
        return dict(bytes=8.0 * (P * (P + 1) // 2), flops=_all_flops(bs))
    if k == "oneint":
        npp = sum(len(a.pexps) * len(b.pexps) for i, a in enumerate(bs.bfs) for b in bs.bfs[:i + 1])
        return dict(bytes=16.0 * n * n, flops=100.0 * npp * nat)
    if k == "xc":
        g = 32 * 194 * nat
        return dict(bytes=8.0 * (g * n + 3 * g + 2 * n * n), flops=3.0 * g * n * n)
    fl = _plan_flops(Ints.get2ints(bs, direct=True).engine)
    if k == "gradient":
        return dict(bytes=8.0 * (2 * n * n + 3 * nat), flops=4.0 * fl)
    mats = {"fock": 2 if case.get("host") else 3, "coulomb": 2, "uhf": 6}[k]
    return dict(bytes=8.0 * mats * n * n, flops=fl)


# ----------------------------------------------------------------- exact --

class _Boys(torch.autograd.Function):
    """F_0 .. F_m(T), stacked first: the top one from the incomplete gamma
    function (its series below T = 1e-3), the others by downward recursion."""

    @staticmethod
    def forward(ctx, T, m):
        top = m + 1   # one more, for the derivative dF_m/dT = -F_{m+1}
        a = top + 0.5
        Ts = T.clamp(min=1e-3)
        big = torch.special.gammainc(torch.full_like(Ts, a), Ts) * (0.5 * math.gamma(a)) * Ts ** (-a)
        small = sum((-T) ** k / (math.factorial(k) * (2 * top + 2 * k + 1)) for k in range(6))
        F = [torch.where(T < 1e-3, small, big)]
        ex = torch.exp(-T)
        for j in range(top - 1, -1, -1):
            F.insert(0, (2 * T * F[0] + ex) / (2 * j + 1))
        ctx.save_for_backward(torch.stack(F[1:]))
        return torch.stack(F[:m + 1])

    @staticmethod
    def backward(ctx, g):
        (up,) = ctx.saved_tensors
        return -(g * up).sum(0), None


def _herm(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _r_integrals(L, alpha, X):
    """R_tuv, t+u+v <= L, of exponent alpha and separation X[..., 3]."""
    F = _Boys.apply(alpha * X.square().sum(-1), L)
    R = {(0, 0, 0): [F[m] * (-2.0 * alpha) ** m for m in range(L + 1)]}
    for n in range(1, L + 1):
        for t, u, v in [x for x in _herm(L) if sum(x) == n]:
            ax = 0 if t else (1 if u else 2)
            c = [t, u, v]
            c[ax] -= 1
            lo = list(c)
            lo[ax] -= 1
            one, two = R[tuple(c)], R.get(tuple(lo))
            R[(t, u, v)] = [X[..., ax] * one[m + 1] + (c[ax] * two[m + 1] if c[ax] else 0.0) for m in range(L + 1 - n)]
    return {k: v[0] for k, v in R.items()}


class _Reference:
    """One- and two-electron integrals of a basis in plain 64-bit torch."""

    def __init__(self, mol, bs):
        f = bs.bfs
        self.n = n = len(f)
        self.Z = torch.tensor([float(a.atno) for a in mol.atoms], dtype=F64, device=DEV)
        self.R = torch.tensor([a.pos() for a in mol.atoms], dtype=F64, device=DEV)
        nprim = np.array([len(b.pexps) for b in f])
        off = np.concatenate([[0], np.cumsum(nprim)])
        ex = np.concatenate([np.asarray(b.pexps, dtype=np.float64) for b in f])
        w = np.concatenate([b.norm * np.asarray(b.pcoefs) * np.asarray(b.pnorms) for b in f])
        fun = np.repeat(np.arange(n), nprim)
        pw = np.array([b.powers for b in f])
        i, j = np.tril_indices(n)
        # every primitive pair of every function pair i >= j
        cnt = nprim[i] * nprim[j]
        pair = np.repeat(np.arange(len(i)), cnt)
        k = np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt)
        p, q = off[i[pair]] + k // nprim[j[pair]], off[j[pair]] + k % nprim[j[pair]]
        put = lambda x, t=F64: torch.as_tensor(np.ascontiguousarray(x), device=DEV).to(t)  # noqa: E731
        self.pair, self.npair = put(pair, torch.int64), len(i)
        self.i, self.j = put(i, torch.int64), put(j, torch.int64)
        self.a, self.b, self.w = put(ex[p]), put(ex[q]), put(w[p] * w[q])
        self.pi, self.pj = put(pw[fun[p]], torch.int64), put(pw[fun[q]], torch.int64)
        atom = np.array([b.atid for b in f])
        self.ai, self.aj = put(atom[fun[p]], torch.int64), put(atom[fun[q]], torch.int64)
        self.L = (self.pi + self.pj).sum(1)

    def _geometry(self, R):
        A, B = R[self.ai], R[self.aj]
        p = self.a + self.b
        return A, B, p, (self.a[:, None] * A + self.b[:, None] * B) / p[:, None]

    def _hermite(self, R, extra):
        """E[axis][i][j][t] (tensors over the primitive pairs) for i <= 2 and
        j <= 2 + extra, the Gaussian product factor included."""
        A, B, p, P = self._geometry(R)
        mu, h = self.a * self.b / p, 0.5 / p
        out = []
        for x in range(3):
            PA, PB = P[:, x] - A[:, x], P[:, x] - B[:, x]
            E = {(0, 0): [torch.exp(-mu * (A[:, x] - B[:, x]) ** 2)]}

            def up(e, d):
                get = lambda t: e[t] if 0 <= t < len(e) else 0.0  # noqa: E731
                return [h * get(t - 1) + d * get(t) + (t + 1) * get(t + 1) for t in range(len(e) + 1)]
            for i in range(3):
                if i:
                    E[(i, 0)] = up(E[(i - 1, 0)], PA)
                for j in range(1, 3 + extra):
                    E[(i, j)] = up(E[(i, j - 1)], PB)
            out.append(E)
        return out

    @staticmethod
    def _pick(E, x, i, j, t, sel_i, sel_j):
        """E[x][i][j][t] per primitive pair, i and j read from the powers."""
        zero = torch.zeros_like(E[x][(0, 0)][0])
        rows = [(E[x][(a, b)][t] if t <= a + b else zero) for a, b in itertools.product(i, j)]
        at = sel_i * len(j) + sel_j
        return torch.stack(rows).gather(0, at[None, :])[0]

    def _hermite_vectors(self, R):
        """[(index of the primitive pairs with L, h[pairs, tuv])] per L."""
        E = self._hermite(R, 0)
        ij = list(range(3))
        one = [[self._pick(E, x, ij, ij, t, self.pi[:, x], self.pj[:, x]) for t in range(5)] for x in range(3)]
        out = []
        for L in range(int(self.L.max()) + 1):
            idx = torch.nonzero(self.L == L)[:, 0]
            if len(idx):
                h = [self.w[idx] * one[0][t][idx] * one[1][u][idx] * one[2][v][idx] for t, u, v in _herm(L)]
                out.append((L, idx, torch.stack(h, 1)))
        return out

    def _square(self, v):
        """Function-pair values to a symmetric matrix."""
        flat = torch.zeros(self.npair, dtype=F64, device=DEV).index_add(0, self.pair, v)
        M = torch.zeros(self.n, self.n, dtype=F64, device=DEV).index_put((self.i, self.j), flat)
        return M + torch.tril(M, -1).T

    def one_electron(self, R):
        _, _, p, P = self._geometry(R)
        E = self._hermite(R, 2)
        ii, jj = list(range(3)), list(range(5))
        s = [[self._pick(E, x, ii, jj, 0, self.pi[:, x], (self.pj[:, x] + d).clamp(min=0)) for d in (-2, 0, 2)] for x in range(3)]
        pre = self.w * (math.pi / p) ** 1.5
        b = self.b
        T = 0.0
        for x in range(3):
            l = self.pj[:, x].to(F64)
            t = -0.5 * (l * (l - 1) * s[x][0] - 2 * b * (2 * l + 1) * s[x][1] + 4 * b * b * s[x][2])
            T = T + t * s[(x + 1) % 3][1] * s[(x + 2) % 3][1]
        V = torch.zeros_like(p)
        for L, idx, h in self._hermite_vectors(R):
            for c0 in range(0, len(idx), 1 << 16):
                at, hc = idx[c0:c0 + (1 << 16)], h[c0:c0 + (1 << 16)]
                Rt = _r_integrals(L, p[at][:, None], P[at][:, None, :] - R[None, :, :])
                v = sum(hc[:, m] * (Rt[k] @ self.Z) for m, k in enumerate(_herm(L)))
                V = V.index_add(0, at, -2.0 * math.pi / p[at] * v)
        return self._square(pre * s[0][1] * s[1][1] * s[2][1]), self._square(pre * T), self._square(V)

    def two_electron(self, R):
        """(ij|kl) as a matrix over the function pairs."""
        _, _, p, P = self._geometry(R)
        out = torch.zeros(self.npair, self.npair, dtype=F64, device=DEV)
        H = self._hermite_vectors(R)
        for (L1, i1, h1), (L2, i2, h2) in itertools.product(H, H):
            if L1 < L2:
                continue
            step = max(1, (1 << 22) // len(i2))
            k1, k2 = _herm(L1), _herm(L2)
            for c0 in range(0, len(i1), step):
                at, hb = i1[c0:c0 + step], h1[c0:c0 + step]
                p1, p2 = p[at][:, None], p[i2][None, :]
                Rt = _r_integrals(L1 + L2, p1 * p2 / (p1 + p2), P[at][:, None, :] - P[i2][None, :, :])
                v = 0.0
                for m, a in enumerate(k1):
                    w = 0.0
                    for n, c in enumerate(k2):
                        w = w + (h2[:, n] * (-1.0) ** sum(c))[None, :] * Rt[tuple(x + y for x, y in zip(a, c))]
                    v = v + hb[:, m][:, None] * w
                v = v * (2.0 * math.pi ** 2.5) / (p1 * p2 * torch.sqrt(p1 + p2))
                cols = torch.zeros(len(at), self.npair, dtype=F64, device=DEV).index_add(1, self.pair[i2], v)
                rows = torch.zeros_like(out).index_add(0, self.pair[at], cols) if out.requires_grad or R.requires_grad else None
                if rows is not None:
                    out = out + rows + (rows.T if L1 > L2 else 0.0)
                else:
                    out.index_add_(0, self.pair[at], cols)
                    if L1 > L2:
                        out.index_add_(1, self.pair[at], cols.T)
        return out

    def dense(self, M):
        full = torch.zeros(self.n, self.n, dtype=torch.int64, device=DEV)
        full[self.i, self.j] = torch.arange(self.npair, device=DEV)
        full = torch.maximum(full, full.T).reshape(-1)
        return M.index_select(0, full).index_select(1, full).reshape((self.n,) * 4)

    def jk(self, M, D):
        I = self.dense(M)
        return torch.einsum("ijkl,kl->ij", I, D), torch.einsum("ikjl,kl->ij", I, D)


def _exact_gradient(mol, bs):
    C, e = _guess(mol, bs)
    D, W = C @ C.T, (C * e) @ C.T
    ref = _Reference(mol, bs)
    R = ref.R.clone().requires_grad_(True)
    S, T, V = ref.one_electron(R)
    J, K = ref.jk(ref.two_electron(R), D)
    i, j = torch.tril_indices(len(R), len(R), -1, device=DEV)
    nuc = (ref.Z[i] * ref.Z[j] / (R[i] - R[j]).norm(dim=1)).sum() if len(i) else 0.0
    energy = 2 * (D * (T + V)).sum() + (D * (2 * J - K)).sum() - 2 * (W * S).sum() + nuc
    return torch.autograd.grad(energy, R)[0].cpu().numpy()


def exact(case, seed):
    k = case["kind"]
    if k in ("stored", "mp2"):
        n = case["nbf"]
        b = _three_index(n, seed)
        B = torch.zeros(b.shape[0], n, n, dtype=F64, device=DEV)
        i, j = torch.tril_indices(n, n, device=DEV)
        B[:, i, j] = b
        B[:, j, i] = b
        if k == "stored":
            D = _stored_density(n, seed)
            J = torch.einsum("qij,q->ij", B, (B * D).sum((1, 2)))
            return 2 * J - torch.einsum("qij,qjk->ik", B @ D, B)
        o = case["nocc"]
        C, e = _orbitals(n, o, seed)
        X = (C[:, :o].T @ B @ C[:, o:]).reshape(b.shape[0], -1)
        V = (X.T @ X).reshape(o, n - o, o, n - o)
        den = e[:o, None, None, None] - e[None, o:, None, None] + e[None, None, :o, None] - e[None, None, None, o:]
        return float((V * (2 * V - V.permute(0, 3, 2, 1)) / den).sum())
    if k in ("xc", "batch"):
        return None   # the grid's and the SCF's own convergence stand behind these
    mol, bs = _basis(case, seed)
    n = len(bs)
    if k == "oneint":
        ref = _Reference(mol, bs)
        S, T, V = ref.one_electron(ref.R)
        return S.cpu().numpy(), (T + V).cpu().numpy()
    if n > (30 if k == "gradient" else 60):
        return None
    if k == "gradient":
        return _exact_gradient(mol, bs)
    ref = _Reference(mol, bs)
    M = ref.two_electron(ref.R)
    if k == "ints":
        return M[torch.tril(torch.ones_like(M, dtype=torch.bool))]
    C, _ = _guess(mol, bs)
    D = C @ C.T
    J, K = ref.jk(M, D)
    if k == "coulomb":
        return J
    if k == "uhf":
        Cb = C[:, :max(1, C.shape[1] - 1)]
        Jb, Kb = ref.jk(M, Cb @ Cb.T)
        return J, Jb, K, Kb
    return (2 * J - K).cpu().numpy() if case["host"] else (J, K)
