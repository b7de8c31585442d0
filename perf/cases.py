"""The work that users of hfsolver_gb300 have it do, as cases that can be timed.

A case is a dict with a "kind":

* rhf      one molecule through hf.rhf: energies, orbitals, MBPT2
* grad     one hf.rhf_gradient call, a force evaluation of molecular dynamics
* batch    many molecules of uneven size in one hf.rhf_batch call
* ints     hf.getInts, the packed integrals of a basis given as arrays
* jk       hf.jk, J and K of a density for such a basis
* transform  hf.transform_int2, packed AO integrals to packed MO integrals

Molecules are clusters of 1 to 16 waters in 6-31G** (25 to 400 functions) as
the tests and bench.py build them, each atom displaced a little at random
("jitter", in A), so that no two seeds give the same geometry, in a cube of
"stretch" times the edge that gives 8 waters in 8 A (a looser cluster keeps
fewer integrals).  The "options" of a case name one of the option sets of
OPTIONS.  Everything a call takes and returns is host memory,
so the inputs are host arrays.

exact() evaluates the same quantities in plain torch in 64 bits, with the
electron repulsion integrals by Gauss-Legendre quadrature of
F_0(T) = int_0^1 exp(-T s^2) ds over the Hermite expansion of each primitive
pair, for the cases small enough for that.
"""
import math

import numpy as np
import torch

import hfsolver_gb300 as hf
from hfsolver_gb300.clusters import water_cluster

NBF_WATER = 25
NOCC_WATER = 5

# option sets of the molecule calls
OPTIONS = {
    # the reference program's own choices: start from the core Hamiltonian, linear
    # mixing, no screening, everything in FP64
    "reference": dict(nscf=100, tolE=1e-12, tolP=1e-10),
    # direct SCF with Schwarz screening and DIIS, an eigensolve per iteration, FP64 MBPT2
    "diis": dict(nscf=100, diis=True, schwarz=1e-12),
    # throughput settings: density purification, incremental Fock builds, atomic
    # start, MBPT2 on the tensor cores
    "fast": dict(nscf=100, diis=True, schwarz=1e-12, purify=True, incremental=True, guess="sad", mp2="split_bf16"),
    # the same with the kernel shapes timed on first use, as bench.py runs it
    "fast_tuned": dict(nscf=60, diis=True, schwarz=1e-12, purify=True, incremental=True, guess="sad",
                       mp2="split_bf16", autotune=True),
    # forces for molecular dynamics: tightly converged, no MBPT2
    "forces": dict(nscf=100, diis=True, schwarz=1e-12, tolP=1e-10, mp2="none"),
}


def listed():
    cases = [
        # one molecule with the reference's settings: every kernel is tiny, launches and waits decide
        {"name": "rhf_w1_reference", "kind": "rhf", "waters": 1, "options": "reference"},
        # a small cluster at throughput settings (75 functions, an odd size)
        {"name": "rhf_w3_fast", "kind": "rhf", "waters": 3, "options": "fast"},
        # a medium cluster converged with an eigensolve per iteration and plain FP64 MBPT2
        {"name": "rhf_w6_diis", "kind": "rhf", "waters": 6, "options": "diis"},
        # the headline benchmark's molecule (200 functions)
        {"name": "rhf_w8_fast", "kind": "rhf", "waters": 8, "options": "fast_tuned"},
        # the largest benchmark molecule (400 functions, 80 occupied orbitals)
        {"name": "rhf_w16_fast", "kind": "rhf", "waters": 16, "options": "fast"},
        # force evaluations of molecular dynamics, small and large
        {"name": "grad_w2", "kind": "grad", "waters": 2, "options": "forces"},
        {"name": "grad_w9", "kind": "grad", "waters": 9, "options": "forces"},
        # many small frames at once (monomers and dimers)
        {"name": "batch_small", "kind": "batch", "molecules": 48, "wmin": 1, "wmax": 2, "options": "fast"},
        # uneven clusters at once, the batch benchmark's mix
        {"name": "batch_mixed", "kind": "batch", "molecules": 20, "wmin": 1, "wmax": 12, "options": "fast"},
        # a caller with its own SCF: all integrals of a trimer, unscreened
        {"name": "ints_w3", "kind": "ints", "waters": 3},
        # a caller with its own SCF: one screened Coulomb and exchange build
        {"name": "jk_w5", "kind": "jk", "waters": 5, "schwarz": 1e-12},
        # a caller with its own integrals: the whole AO to MO transform in FP64
        {"name": "transform_n100", "kind": "transform", "n": 100},
    ]
    return [c if c["kind"] == "transform" else {**c, "jitter": 0.03, "stretch": 1.0} for c in cases]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["rhf", "rhf", "rhf", "grad", "grad", "batch", "batch", "ints", "jk", "transform"])
    if kind == "transform":
        return {"kind": kind, "n": _log_int(rng, 20, 120)}
    if kind == "rhf":
        options = rng.choice(["fast", "fast", "fast_tuned", "diis", "reference"])
        waters = 1 if options == "reference" else _log_int(rng, 1, 7 if options == "diis" else 16)
        case = {"kind": kind, "waters": waters, "options": options}
    elif kind == "grad":
        case = {"kind": kind, "waters": _log_int(rng, 1, 11), "options": "forces"}
    elif kind == "batch":
        wmin = _log_int(rng, 1, 5)
        wmax = rng.randint(wmin, 12)
        # at most 80 waters in all
        most = max(2, 160 // (wmin + wmax))
        case = {"kind": kind, "molecules": _log_int(rng, 2, min(64, most)), "wmin": wmin, "wmax": wmax,
                "options": "fast"}
    elif kind == "ints":
        case = {"kind": kind, "waters": _log_int(rng, 1, 4)}
    else:
        case = {"kind": kind, "waters": _log_int(rng, 1, 8), "schwarz": rng.choice([0.0, 1e-12, 1e-10])}
    return {**case, "jitter": round(rng.uniform(0.01, 0.05), 3), "stretch": round(rng.uniform(1.0, 1.3), 2)}


# ---------------------------------------------------------------- inputs
def _molecule(case, seed, waters=None):
    # 16 waters in an 11 A cube, other sizes at the density of 8 waters in an 8 A cube
    w = case["waters"] if waters is None else waters
    box = 11.0 if w == 16 else 8.0 * (w / 8.0) ** (1.0 / 3.0)
    return water_cluster(w, box=case["stretch"] * box, seed=seed, jitter=case["jitter"])


# 6-31G** shells (L, exponents, coefficients) of the two elements used
_SHELLS = {
    1: [(0, [18.731137, 2.8253937, 0.6401217], [0.0334946, 0.23472695, 0.81375733]),
        (0, [0.1612778], [1.0]),
        (1, [1.1], [1.0])],
    8: [(0, [5484.6717, 825.23495, 188.04696, 52.9645, 16.89757, 5.7996353],
         [0.0018311, 0.0139501, 0.0684451, 0.2327143, 0.470193, 0.3585209]),
        (0, [15.539616, 3.5999336, 1.0137618], [-0.1107775, -0.1480263, 1.130767]),
        (1, [15.539616, 3.5999336, 1.0137618], [0.0708743, 0.3397528, 0.7271586]),
        (0, [0.2700058], [1.0]),
        (1, [0.2700058], [1.0]),
        (2, [0.8], [1.0])],
}


def _basis(atno, xyz):
    """The Cartesian functions as arrays, the way getInts and jk take them, and each one's atom."""
    def odd(k):  # (2 k - 1)!!
        return math.prod(range(2 * k - 1, 0, -2))

    nprim, centre, power, coef, alpha, atom = [], [], [], [], [], []
    for a, z in enumerate(atno):
        for L, ex, co in _SHELLS[int(z)]:
            for k in range(L + 1):
                for m in range(k + 1):
                    lmn = (L - k, k - m, m)
                    dd = odd(lmn[0]) * odd(lmn[1]) * odd(lmn[2])
                    # the power of two in single precision, as in hfsolver's norm_prim
                    two = float(np.float32(2.0 ** (2 * L + 1.5)))
                    c = [x * math.sqrt(two * e ** (L + 1.5) / dd / math.pi ** 1.5) for x, e in zip(co, ex)]
                    if len(ex) > 1:
                        s = sum(ci * cj * (ei + ej) ** (-L - 1.5) for ci, ei in zip(c, ex) for cj, ej in zip(c, ex))
                        c = [x / math.sqrt(s * dd * math.pi ** 1.5 / 2.0 ** L) for x in c]
                    nprim.append(len(ex))
                    centre.append(xyz[a])
                    power.append(lmn)
                    coef += c
                    alpha += ex
                    atom.append(a)
    nprim = np.array(nprim, dtype=np.int32)
    centre = np.array(centre)
    power = np.array(power, dtype=np.int32)
    istart = np.concatenate([[0], np.cumsum(nprim)[:-1]]).astype(np.int32)
    args = [nprim, istart] + [np.ascontiguousarray(centre[:, k]) for k in range(3)]
    args += [np.ascontiguousarray(power[:, k]) for k in range(3)] + [np.array(coef), np.array(alpha)]
    return args, np.array(atom)


def _density(n, nocc, seed):
    """2 C C^T of random orthonormal orbitals."""
    q = np.linalg.qr(np.random.default_rng(seed).standard_normal((n, nocc)))[0]
    return 2.0 * q @ q.T


def _integrals(n, seed):
    """A packed array with the symmetry, the sign structure and the decay of two-electron
    integrals, sum_Q B_Q,ij B_Q,kl with B local in i - j, and an orthogonal matrix."""
    rng = np.random.default_rng(seed)
    m = n * (n + 1) // 2
    i, j = np.tril_indices(n)
    B = rng.standard_normal((m, n)) * np.exp(-0.15 * (i - j))[:, None] * np.exp(rng.normal(-1.0, 1.0, n))[None, :]
    B = torch.from_numpy(B)
    if torch.cuda.is_available():
        B = B.cuda()
    M = B @ B.T
    a = torch.ones(m, m, dtype=torch.bool, device=B.device).tril_()
    packed = M[a].cpu().numpy()
    return packed, np.linalg.qr(rng.standard_normal((n, n)))[0]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("rhf", "grad"):
        atno, xyz = _molecule(case, seed)
        return {"kind": kind, "atno": atno, "xyz": xyz, "options": hf.RHFOptions(**OPTIONS[case["options"]])}
    if kind == "batch":
        # spread evenly over the range, so that every seed has the same amount of work
        sizes = np.round(np.linspace(case["wmin"], case["wmax"], case["molecules"])).astype(int)
        mols = [_molecule(case, seed * 1000 + 7 * k + 1, int(s)) for k, s in enumerate(sizes)]
        return {"kind": kind, "molecules": mols, "options": hf.RHFOptions(**OPTIONS[case["options"]])}
    if kind == "ints":
        return {"kind": kind, "basis": _basis(*_molecule(case, seed))[0]}
    if kind == "jk":
        args, _ = _basis(*_molecule(case, seed))
        n = len(args[0])
        return {"kind": kind, "basis": args, "P": _density(n, NOCC_WATER * case["waters"], seed),
                "schwarz": case["schwarz"]}
    int2, C = _integrals(case["n"], seed)
    return {"kind": kind, "int2": int2, "C": C}


ENERGIES = ("Etot", "E0", "Enuc", "Ekin", "E2")


def run(state):
    kind = state["kind"]
    if kind == "rhf":
        r = hf.rhf(state["atno"], state["xyz"], state["options"], want_orbitals=True)
        # the orbitals are fixed up to their signs: what is compared is the density they make
        occ = r["C"][:, :r["nocc"]]
        out = {k: r[k] for k in ENERGIES}
        out["lam"], out["P"] = r["lam"], 2.0 * occ @ occ.T
        return out
    if kind == "grad":
        r, g = hf.rhf_gradient(state["atno"], state["xyz"], state["options"])
        return {"Etot": r["Etot"], "grad": g}
    if kind == "batch":
        rs = hf.rhf_batch(state["molecules"], state["options"])
        return {k: np.array([r[k] for r in rs]) for k in ENERGIES}
    if kind == "ints":
        return hf.getInts(*state["basis"])
    if kind == "jk":
        J, K = hf.jk(*state["basis"], state["P"], state["schwarz"])
        return {"J": J, "K": K}
    return hf.transform_int2(state["int2"], state["C"])


# ---------------------------------------------------------------- work
def _packed(n):
    m = n * (n + 1) // 2
    return m * (m + 1) // 2


def _rhf_flops(waters, mp2, gradient=False):
    """Integrals once (about 300 operations for each of the distinct ones that survive
    screening in a cluster of this density), 10 Fock builds of 12 operations an
    integral and 10 densities of 4 n^3, and the MBPT2 half transform."""
    n, o = NBF_WATER * waters, NOCC_WATER * waters
    v = n - o
    kept = _packed(n) * min(1.0, 6.0 / waters)
    f = kept * (300 + 120) + 40.0 * n ** 3
    if mp2:
        f += o * n ** 4 + o * v * n ** 3 + 2.0 * o * o * v * n * n + 2.0 * o * o * v * v * n
    if gradient:
        f += kept * 1500
    return f


def work(case):
    kind = case["kind"]
    if kind in ("rhf", "grad"):
        w = case["waters"]
        n = NBF_WATER * w
        out = 8 * (n * n + n + 5) if kind == "rhf" else 8 * 9 * w
        return {"bytes": 3 * w * 28 + out, "flops": _rhf_flops(w, kind == "rhf", kind == "grad")}
    if kind == "batch":
        ws = np.linspace(case["wmin"], case["wmax"], case["molecules"])
        return {"bytes": float(sum(84 * w + 40 for w in ws)), "flops": float(sum(_rhf_flops(w, True) for w in ws))}
    if kind == "ints":
        n = NBF_WATER * case["waters"]
        return {"bytes": 8 * _packed(n), "flops": 300.0 * _packed(n)}
    if kind == "jk":
        n = NBF_WATER * case["waters"]
        return {"bytes": 3 * 8 * n * n, "flops": 312.0 * _packed(n) * min(1.0, 6.0 / case["waters"])}
    n = case["n"]
    return {"bytes": 16 * _packed(n) + 8 * n * n, "flops": 4.0 * n ** 5}


# ---------------------------------------------------------------- the same in plain torch
class _Exact:
    """Integrals of a function list (args, atom) by the definitions, on `device`."""

    def __init__(self, args, atom, atno, xyz, device):
        nprim, _, _, _, _, lp, mp, npw, coef, alpha = args
        self.n, self.dev = len(nprim), device
        f = np.repeat(np.arange(self.n), nprim)
        pw = np.stack([lp, mp, npw], 1)[f]
        i, j = np.nonzero(f[:, None] >= f[None, :])
        self.fij = torch.as_tensor(f[i] * (f[i] + 1) // 2 + f[j], device=device)
        self.m = self.n * (self.n + 1) // 2
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=device)  # noqa: E731
        self.a, self.b, self.cc = t(alpha[i]), t(alpha[j]), t(coef[i] * coef[j])
        self.pi, self.pj = torch.as_tensor(pw[i], device=device), torch.as_tensor(pw[j], device=device)
        self.ai, self.aj = torch.as_tensor(atom[f[i]], device=device), torch.as_tensor(atom[f[j]], device=device)
        self.atno, self.xyz = t(np.asarray(atno, float)), t(xyz)
        x, w = np.polynomial.legendre.leggauss(48)
        self.x, self.w = t((x + 1) / 2), t(w / 2)

    def pairs(self, xyz, jmax=2):
        """p, P and the Hermite coefficients E[i][j] (pairs, 3, i + j + 1 padded to 7) of every primitive pair."""
        A, B = xyz[self.ai], xyz[self.aj]
        p = self.a + self.b
        P = (self.a[:, None] * A + self.b[:, None] * B) / p[:, None]
        h = (0.5 / p)[:, None, None]
        t1 = torch.arange(1, 7, device=self.dev, dtype=torch.float64)
        zero = torch.zeros(p.shape[0], 3, 1, dtype=torch.float64, device=self.dev)

        def up(E, d):
            low = torch.cat([zero, E[..., :-1]], -1)
            high = torch.cat([E[..., 1:] * t1, zero], -1)
            return h * low + d[..., None] * E + high

        E0 = torch.exp(-(self.a * self.b / p)[:, None] * (A - B) ** 2)[..., None]
        E = [[torch.cat([E0] + [zero] * 6, -1)]]
        for i in range(2):
            E.append([up(E[i][0], P - A)])
        for i in range(3):
            for j in range(jmax):
                E[i].append(up(E[i][j], P - B))
        return p, P, E

    def pick(self, E, dj=0):
        """The Hermite coefficients of each pair for its own powers, the second raised by dj (zero below 0)."""
        tab = torch.stack([torch.stack(r, 0) for r in E], 0)  # (3, jmax + 1, pairs, 3, 7)
        j = self.pj + dj
        k = torch.arange(j.shape[0], device=self.dev)[:, None]
        d = torch.arange(3, device=self.dev)[None, :]
        return tab[self.pi, j.clamp(0, tab.shape[1] - 1), k, d] * (j >= 0)[..., None]

    def fold(self, v):
        """Sum of the primitive pairs' values into the symmetric matrix of the functions."""
        tri = torch.zeros(self.m, dtype=torch.float64, device=self.dev).index_add(0, self.fij, v * self.cc)
        return self.square(tri)

    def square(self, tri):
        i, j = torch.tril_indices(self.n, self.n, device=self.dev)
        M = torch.zeros(self.n, self.n, dtype=torch.float64, device=self.dev)
        return M.index_put((i, j), tri).index_put((j, i), tri)

    @staticmethod
    def hermite(a, X, top):
        """d^k/dX^k exp(-a X^2), k = 0 .. top."""
        D = [torch.exp(-a * X * X)]
        for k in range(top):
            D.append(-2 * a * (X * D[k] + (k * D[k - 1] if k else 0)))
        return D

    def one_electron(self, xyz):
        p, P, E = self.pairs(xyz, 4)
        e0, ep, em = self.pick(E)[..., 0], self.pick(E, 2)[..., 0], self.pick(E, -2)[..., 0]
        q = (math.pi / p) ** 1.5
        S = q * e0.prod(1)
        b, j = self.b, self.pj.double()
        T = b * (2 * j.sum(1) + 3) * S
        for d in range(3):
            o = [k for k in range(3) if k != d]
            rest = q * e0[:, o[0]] * e0[:, o[1]]
            T = T - 2 * b * b * rest * ep[:, d] - 0.5 * j[:, d] * (j[:, d] - 1) * rest * em[:, d]
        e = self.pick(E)
        X = P[:, None, :] - xyz[None, :, :]
        T0 = p[:, None] * (X * X).sum(-1)
        s = torch.sqrt(45.0 / T0.clamp_min(45.0))
        V = torch.zeros_like(p)
        for x, w in zip(self.x, self.w):
            D = self.hermite((p[:, None] * (s * x) ** 2)[..., None], X, 4)
            v = sum(e[:, None, :, t] * D[t] for t in range(5)).prod(-1)
            V = V - (self.atno[None, :] * w * s * v).sum(1)
        return self.fold(S), self.fold(T), self.fold(V * 2 * math.pi / p)

    def chunks(self, size):
        n = self.cc.shape[0]
        step = max(1, size // (48 * n))
        return [(k, min(n, k + step)) for k in range(0, n, step)]

    def rows(self, r0, r1, p, P, e):
        """The integrals of primitive pairs r0 .. r1 - 1 with all pairs, contracted over the second: (r, m)."""
        pa, pb = p[r0:r1, None], p[None, :]
        al = pa * pb / (pa + pb)
        X = P[r0:r1, None, :] - P[None, :, :]
        s = torch.sqrt(45.0 / (al * (X * X).sum(-1)).clamp_min(45.0))
        a = al[..., None] * (s[..., None] * self.x) ** 2
        v = s[..., None] * self.w
        # the highest Hermite orders on each side
        for d in range(3):
            ta = int((self.pi + self.pj)[r0:r1, d].max())
            D = self.hermite(a, X[..., d, None], ta + 4)
            tot = None
            for t in range(ta + 1):
                y = sum((-1.0) ** u * e[None, :, d, u, None] * D[t + u] for u in range(5))
                y = y * e[r0:r1, None, d, t, None]
                tot = y if tot is None else tot + y
            v = v * tot
        v = v.sum(-1) * (2 * math.pi ** 2.5) / (pa * pb * torch.sqrt(pa + pb)) * self.cc[r0:r1, None] * self.cc[None, :]
        return torch.zeros(r1 - r0, self.m, dtype=torch.float64, device=self.dev).index_add(1, self.fij, v)

    def eri(self):
        """(ij|kl) over function pairs, (m, m)."""
        p, P, E = self.pairs(self.xyz)
        e = self.pick(E)
        M = torch.zeros(self.m, self.m, dtype=torch.float64, device=self.dev)
        for r0, r1 in self.chunks(1 << 23):
            M.index_add_(0, self.fij[r0:r1], self.rows(r0, r1, p, P, e))
        return M

    def unpack(self, M):
        """(i, j, k, l) of the pair matrix."""
        i, j = torch.meshgrid(*[torch.arange(self.n, device=self.dev)] * 2, indexing="ij")
        hi, lo = torch.maximum(i, j), torch.minimum(i, j)
        t = (hi * (hi + 1) // 2 + lo).reshape(-1)
        return M[t][:, t].reshape(self.n, self.n, self.n, self.n)

    def repulsion(self, xyz):
        d = (xyz[:, None, :] - xyz[None, :, :]).pow(2).sum(-1) + torch.eye(len(xyz), dtype=torch.float64, device=self.dev)
        z = self.atno[:, None] * self.atno[None, :]
        return 0.5 * (z / d.sqrt()).sum() - 0.5 * torch.diagonal(z).sum()


def _scf(x, nocc):
    """Converged closed-shell RHF: energies, orbitals and what made them."""
    S, T, V = x.one_electron(x.xyz)
    I = x.unpack(x.eri())
    H = T + V
    s, U = torch.linalg.eigh(S)
    X = U / s.sqrt()
    F, Fs, es = H, [], []
    for it in range(200):
        lam, C = torch.linalg.eigh(X.T @ F @ X)
        C = X @ C
        P = 2 * C[:, :nocc] @ C[:, :nocc].T
        F = H + torch.einsum("ijkl,kl->ij", I, P) - 0.5 * torch.einsum("ikjl,kl->ij", I, P)
        E0 = 0.5 * float((P * (H + F)).sum())
        err = X.T @ (F @ P @ S - S @ P @ F) @ X
        if float(err.abs().max()) < 1e-12 * len(S) ** 0.5:
            break
        Fs, es = (Fs + [F])[-8:], (es + [err])[-8:]
        k = len(Fs)
        B = torch.zeros(k + 1, k + 1, dtype=torch.float64, device=x.dev)
        B[:k, :k] = torch.stack([torch.stack([(u * w).sum() for w in es]) for u in es])
        B[:k, :k] /= B[:k, :k].diagonal().max()
        B[k, :k] = B[:k, k] = -1
        r = torch.zeros(k + 1, dtype=torch.float64, device=x.dev)
        r[k] = -1
        c = torch.linalg.lstsq(B.cpu(), r.cpu()[:, None], driver="gelsd").solution.reshape(-1).to(x.dev)[:k]
        F = sum(ci * Fi for ci, Fi in zip(c, Fs))
    lam, C = torch.linalg.eigh(X.T @ F @ X)
    C = X @ C
    return {"E0": E0, "lam": lam, "C": C, "P": P, "I": I, "Ekin": float((P * T).sum()), "Enuc": float(x.repulsion(x.xyz))}


def _mp2(r, nocc):
    C, lam = r["C"], r["lam"]
    t = torch.einsum("ijkl,ia->ajkl", r["I"], C[:, :nocc])
    t = torch.einsum("ajkl,jr->arkl", t, C[:, nocc:])
    t = torch.einsum("arkl,kb->arbl", t, C[:, :nocc])
    t = torch.einsum("arbl,ls->arbs", t, C[:, nocc:])
    o, v = lam[:nocc], lam[nocc:]
    D = o[:, None, None, None] + o[None, None, :, None] - v[None, :, None, None] - v[None, None, None, :]
    return float((t * (2 * t - t.permute(0, 3, 2, 1)) / D).sum())


def _gradient(x, r, nocc):
    """dE/dR with the density and energy-weighted density held fixed, by torch's autograd over the integrals."""
    C, P = r["C"], r["P"]
    W = 2 * (C[:, :nocc] * r["lam"][:nocc]) @ C[:, :nocc].T
    # over function pairs i >= j and k >= l: twice the off-diagonal ones
    i, j = torch.tril_indices(x.n, x.n, device=x.dev)
    two = torch.where(i == j, 1.0, 2.0).double()
    G = 0.5 * P[i, j][:, None] * P[i, j][None, :]
    G -= 0.125 * (P[i][:, i] * P[j][:, j] + P[i][:, j] * P[j][:, i])
    G *= two[:, None] * two[None, :]
    xyz = x.xyz.clone().requires_grad_(True)
    S, T, V = x.one_electron(xyz)
    g = torch.autograd.grad((P * (T + V)).sum() - (W * S).sum() + x.repulsion(xyz), xyz)[0]
    for r0, r1 in x.chunks(1 << 21):
        p, Pc, E = x.pairs(xyz)
        e = x.pick(E)
        g = g + torch.autograd.grad((x.rows(r0, r1, p, Pc, e) * G[x.fij[r0:r1]]).sum(), xyz)[0]
    return g


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "transform":
        s = prepare(case, seed)
        n = case["n"]
        m = n * (n + 1) // 2
        M = torch.zeros(m, m, dtype=torch.float64, device=dev)
        k, l = torch.tril_indices(m, m, device=dev)
        M[k, l] = torch.as_tensor(s["int2"], device=dev)
        M[l, k] = M[k, l]
        i, j = torch.tril_indices(n, n, device=dev)
        C = torch.as_tensor(s["C"], device=dev)
        for _ in range(2):  # both pair indices in turn
            Q = torch.zeros(m, n, n, dtype=torch.float64, device=dev)
            Q[:, i, j] = M
            Q[:, j, i] = M
            M = (C.T @ Q @ C)[:, i, j].T.contiguous()
        return M[k, l].cpu().numpy()
    if kind == "batch" or case["waters"] > (2 if kind == "grad" else 3):
        return None
    atno, xyz = _molecule(case, seed)
    args, atom = _basis(atno, xyz)
    x = _Exact(args, atom, atno, xyz, dev)
    nocc = NOCC_WATER * case["waters"]
    if kind == "ints":
        M = x.eri()
        k, l = torch.tril_indices(x.m, x.m, device=dev)
        return M[k, l].cpu().numpy()
    if kind == "jk":
        I, P = x.unpack(x.eri()), torch.as_tensor(_density(x.n, nocc, seed), device=dev)
        return {"J": torch.einsum("ijkl,kl->ij", I, P).cpu().numpy(),
                "K": torch.einsum("ikjl,kl->ij", I, P).cpu().numpy()}
    r = _scf(x, nocc)
    if kind == "grad":
        return {"Etot": r["E0"] + r["Enuc"], "grad": _gradient(x, r, nocc).cpu().numpy()}
    return {"Etot": r["E0"] + r["Enuc"], "E0": r["E0"], "Enuc": r["Enuc"], "Ekin": r["Ekin"], "E2": _mp2(r, nocc),
            "lam": r["lam"].cpu().numpy(), "P": r["P"].cpu().numpy()}
