"""Performance cases of the library: what an SCF program has it do, by its public entry points.

A case is one call -- a Fock build (from device or host arrays, closed or open shell, plain FP64 or the
mixed FP32/FP64 form, a full density or the small density difference of an incremental build), a Fock build of
many molecules at once, the one-electron integrals of a QM/MM step, or a whole RHF solve -- on a seeded water
cluster or alkane.  ``listed()`` names the cases, ``draw`` makes more of the same ranges.
"""
import math

import numpy as np
import torch

from quick_b200 import autotune, molecules
from quick_b200.basis import build_basis
from quick_b200.get2e import Get2e, Get2eBatch
from quick_b200.scf import RHF, GraphSCF, oei

#: integral cutoff and primitive limit of a production Fock build, and of the small molecules' tight ones
CUT, PRIM = 1e-10, 1e-11


def listed():
    fock = {"kind": "fock", "mol": "water", "cut": CUT, "bound": 0.0, "delta": 0.0, "streams": -1, "merge": False,
            "tune": False}
    return [
        # one water in a minimal basis: the smallest build there is, all launch latency (an atom or a monomer
        # inside a fragment method, each cycle of a small solve)
        dict(fock, name="w1_sto3g", n=1, basis="STO-3G"),
        # four waters in STO-3G (28 functions) at the launch choices that the autotuner makes for such molecules:
        # one merged kernel for the s and p classes, no forked streams
        dict(fock, name="w4_sto3g", n=4, basis="STO-3G", streams=0, merge=True),
        # ten waters in 6-31G* (190 functions) from host arrays: the drop-in call of a program that keeps its
        # matrices on the CPU
        dict(fock, kind="host", name="host_w10_631gs", n=10, basis="6-31G*"),
        # the late cycles of a solve: the same kernels on a small density difference, most of it screened away
        dict(fock, name="delta_w20_631gs", n=20, basis="6-31G*", delta=1e-4, streams=0),
        # the benchmark's headline molecule, 32 waters in 6-31G* (608 functions), tuned as the benchmark tunes it
        dict(fock, name="w32_631gs", n=32, basis="6-31G*", tune=True),
        # the largest: C40H82 in 6-31G** (1010 functions), p functions on every hydrogen, long and thin
        dict(fock, name="c40h82_631gss", mol="alkane", n=40, basis="6-31G**", streams=0),
        # twelve waters in cc-pVTZ (780 functions): long contractions, d and f shells
        dict(fock, name="w12_ccpvtz", n=12, basis="CC-PVTZ", streams=0),
        # the mixed form: quartets under the bound in FP32
        dict(fock, name="mixed_w16_631gss", n=16, basis="6-31G**", bound=1e-5, streams=0),
        # open shell: the doublet cation of three waters, alpha and beta Fock matrices, f shells in a small molecule
        dict(fock, kind="uhf", name="uhf_w3_ccpvtz", n=3, basis="CC-PVTZ"),
        # a serving step: 24 molecules of one to eight waters in one call
        {"kind": "batch", "name": "batch_24_mixed", "count": 24, "n": 8, "cut": CUT},
        # a QM/MM step's set-up: twenty waters and 4000 point charges around them, from and to host arrays
        {"kind": "oei", "name": "oei_w20_4000", "n": 20, "basis": "6-31G*", "charges": 4000},
        # a whole solve, the cycle captured as a CUDA graph, from the SAD guess to 1e-7
        {"kind": "scf", "name": "scf_w6_631gs", "n": 6, "basis": "6-31G*", "cut": CUT},
    ]


def draw(rng):
    def size(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))

    kind = rng.choice(["fock"] * 8 + ["host"] * 2 + ["uhf"] * 2 + ["batch"] * 2 + ["oei"] * 2 + ["scf"] * 2)
    most = {"STO-3G": 40, "6-31G": 36, "6-31G*": 36, "6-31G**": 24, "CC-PVDZ": 24, "CC-PVTZ": 10}
    basis = rng.choice(list(most))
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(6, 32), "n": rng.randint(3, 8), "cut": CUT}
    if kind == "oei":
        basis = rng.choice(["STO-3G", "6-31G*", "6-31G**"])
        return {"kind": kind, "n": size(2, 24), "basis": basis, "charges": rng.choice([0, size(60, 4000)])}
    if kind == "scf":
        return {"kind": kind, "n": size(2, 8), "basis": rng.choice(["STO-3G", "6-31G", "6-31G**", "CC-PVDZ"]),
                "cut": rng.choice([CUT, 1e-9, 1e-11])}
    mol = "alkane" if rng.random() < 0.25 else "water"
    n = size(1, most[basis] // (2 if kind == "uhf" else 1))
    if mol == "alkane":
        n = max(2, min(n, most[basis] // 2))
    case = {"kind": kind, "mol": mol, "n": n, "basis": basis, "cut": rng.choice([CUT, CUT, 1e-9, 1e-11]),
            "bound": 0.0, "delta": 0.0, "streams": 0 if n * len(basis) > 60 else -1, "merge": False, "tune": False}
    if kind == "fock":
        if rng.random() < 0.25:
            case["bound"] = rng.choice([1e-6, 1e-5])
        if rng.random() < 0.3:
            case["delta"] = 10.0 ** rng.uniform(-6, -2)
        if basis == "STO-3G":
            case["merge"] = rng.random() < 0.4
    return case


# ---------------------------------------------------------------- inputs
def _molecule(kind, n, seed):
    if kind == "alkane":
        return molecules.alkane(n, seed=seed)
    return molecules.water_cluster(n, max(6.0, 3.15 * n ** (1.0 / 3.0)), seed=seed)


def _basis(case, seed):
    return build_basis(_molecule(case.get("mol", "water"), case["n"], seed), case["basis"])


def _charges(case, basis, seed):
    """MM point charges (three-site waters' magnitudes) in a shell around the molecule, at least 2 A from it."""
    m = case["charges"]
    if m == 0:
        return None
    rng = np.random.default_rng(seed + 17)
    xyz = basis.mol.xyz
    c = xyz.mean(axis=0)
    out = np.zeros((0, 3))
    while len(out) < m:
        v = rng.normal(size=(2 * m, 3))
        v *= (28.0 * rng.random((2 * m, 1)) ** (1 / 3)) / np.linalg.norm(v, axis=1, keepdims=True)
        v += c
        far = np.sqrt(((v[:, None, :] - xyz[None]) ** 2).sum(-1)).min(1) > 3.8
        out = np.concatenate([out, v[far]])
    q = np.where(np.arange(m) % 3 == 0, -0.834, 0.417)
    return out[:m], q


def _symmetric(D):
    return 0.5 * (D + D.T)


def _density(rhf, case, seed):
    """The density of the generalised Wolfsberg-Helmholz guess, or a small difference of such a density."""
    D = _symmetric(rhf.guess("gwh"))
    if case["delta"]:
        g = torch.Generator(device=D.device).manual_seed(seed)
        noise = torch.randn(D.shape, generator=g, dtype=D.dtype, device=D.device)
        D = case["delta"] * _symmetric(D * noise)
    return D


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        engines, Ds = [], []
        for k in range(case["count"]):
            c = {"n": 1 + 5 * k % case["n"], "basis": "STO-3G" if k % 2 else "6-31G*", "delta": 0.0}
            b = _basis(c, seed * 64 + k)
            eng = Get2e(b, integral_cutoff=case["cut"], prim_limit=0.1 * case["cut"])
            Ds.append(_density(RHF(b, engine=eng), c, seed))
            eng.prepare()
            engines.append(eng)
        return {"kind": kind, "batch": Get2eBatch(), "engines": engines, "D": Ds}
    b = _basis(case, seed)
    if kind == "oei":
        return {"kind": kind, "basis": b, "ext": _charges(case, b, seed)}
    if kind == "scf":
        return {"kind": kind, "scf": GraphSCF(RHF(b, integral_cutoff=case["cut"]))}
    eng = Get2e(b, integral_cutoff=case["cut"], prim_limit=0.1 * case["cut"])
    if case["bound"]:
        eng.set_precision(case["bound"])
    if case["streams"] >= 0:
        eng.set_streams(case["streams"])
    if case["merge"]:
        eng.set_merge_sp(True)
    rhf = RHF(b, engine=eng)
    st = {"kind": kind, "eng": eng}
    if kind == "uhf":
        ne = b.mol.nelec - 1 + b.mol.nelec % 2   # an odd electron count
        rhf.nocc = (ne + 1) // 2
        st["Da"] = 0.5 * _density(rhf, case, seed)
        rhf.nocc = ne // 2
        st["Db"] = 0.5 * _density(rhf, case, seed)
    else:
        st["D"] = _density(rhf, case, seed)
        if kind == "host":
            st["D"] = st["D"].cpu().numpy()
    if case["tune"]:
        autotune.tune(eng, st["D"], reps=2)
    eng.prepare()
    return st


def run(st):
    kind = st["kind"]
    if kind == "fock":
        return st["eng"].fock2e(st["D"])
    if kind == "host":
        return st["eng"].fock2e_host(st["D"])
    if kind == "uhf":
        return st["eng"].fock2e_uhf(st["Da"], st["Db"])
    if kind == "batch":
        return st["batch"].fock2e(st["engines"], st["D"])
    if kind == "oei":
        return oei(st["basis"], st["ext"])
    r = st["scf"].run(denserms=1e-7)
    return {"E": r["E"], "D": r["D"], "F": r["F"]}


def tolerance(case):
    """Everything is 64-bit: a sum in another order moves a Fock matrix by about 1e-14 of its norm, and what the screens
    leave out is 1e-11 to 7e-11 of it (against ``exact``), more where the density is a small difference; the mixed
    form's small quartets carry FP32's rounding; a solve stops at a density change of 1e-7."""
    if case["kind"] == "scf":
        return {"rel": 1e-8, "max": 1e-6}
    if case["kind"] == "oei":
        return {"rel": 1e-12, "max": 1e-10}
    if case.get("delta"):
        return {"rel": max(1e-9, 1e-2 * case["cut"] / case["delta"]), "max": max(1e-7, case["cut"] / case["delta"])}
    if case.get("bound"):
        return {"rel": 1e-9, "max": 1e-7}
    return {"rel": 1e-10, "max": 1e-8}


# ---------------------------------------------------------------- work
def _shells(b):
    """(centre, L, exponents, coefficients, first function, per-function factors) of every s, p, d and f shell."""
    out = []
    for s in range(b.nshell):
        k, f = int(b.kprim[s]), int(b.ksumtype[s]) - 1
        for L in range(int(b.qstart[s]), int(b.qfinal[s]) + 1):
            f0 = f + int(b.qsbasis[s, L])
            n = (L + 1) * (L + 2) // 2
            out.append((b.xyz[int(b.katom[s]) - 1], L, b.gcexpo[:k, f + L], b.gccoeff[:k, f + L], f0,
                        b.cons[f0:f0 + n], [tuple(int(x) for x in b.klmn[:, i]) for i in range(f0, f0 + n)]))
    return out


def _nherm(L):
    return (L + 1) * (L + 2) * (L + 3) // 6


def _fock_work(b, cut):
    """Bytes and operations of one build: the shell and primitive quartets above the cutoffs by the (ss|ss) estimate of
    their bounds; a primitive quartet costs its Boys function and one multiply-add per pair of intermediates and
    recursion term, a quartet twelve operations per integral."""
    groups = {}
    sh = _shells(b)
    nprim_pairs = 0
    for i, (A, La, ea, ca, *_) in enumerate(sh):
        for B, Lb, eb, cb, *_ in sh[:i + 1]:
            p = ea[:, None] + eb[None]
            r2 = float(((A - B) ** 2).sum())
            y = np.abs(ca[:, None] * cb[None]) * np.exp(-ea[:, None] * eb[None] / p * r2) * np.sqrt(
                34.98683665524972 / (p * p * np.sqrt(2 * p))) / np.sqrt(p) ** (La + Lb) / 2.0 ** (La + Lb)
            if y.sum() < 0.1 * cut:
                continue
            nprim_pairs += y.size
            g = groups.setdefault((La + Lb, La, Lb), ([], []))
            g[0].append(y.sum())
            g[1].append(y.ravel())
    rec = [(L, La, Lb, np.sort(np.array(y)), np.sort(np.concatenate(yp))) for (L, La, Lb), (y, yp) in groups.items()]

    def above(x, y, limit):
        return float((len(y) - np.searchsorted(y, limit / np.maximum(x, 1e-300))).sum())

    def ncart(L):
        return (L + 1) * (L + 2) // 2

    flops = 0.0
    for i, (L1, a1, b1, y1, p1) in enumerate(rec):
        for j, (L2, a2, b2, y2, p2) in enumerate(rec[:i + 1]):
            half = 0.5 if i == j else 1.0
            ne = _nherm(L1) - (_nherm(a1 - 1) if a1 else 0) if a1 >= b1 else _nherm(L1) - (_nherm(b1 - 1) if b1 else 0)
            nf = _nherm(L2) - (_nherm(a2 - 1) if a2 else 0) if a2 >= b2 else _nherm(L2) - (_nherm(b2 - 1) if b2 else 0)
            flops += half * above(p1, p2, 0.1 * cut) * (50 + 8 * (L1 + L2) + (10 * ne * nf if L1 + L2 else 0))
            flops += half * above(y1, y2, cut) * 12 * ncart(a1) * ncart(b1) * ncart(a2) * ncart(b2)
    return 16.0 * b.nbasis ** 2 + 80.0 * nprim_pairs, flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        each = [_fock_work(_basis({"n": 1 + 5 * k % case["n"], "basis": "STO-3G" if k % 2 else "6-31G*"}, k), CUT)
                for k in range(case["count"])]
        return {"bytes": sum(e[0] for e in each), "flops": sum(e[1] for e in each)}
    b = _basis(case, 1)
    if kind == "oei":
        prims = [(L, len(e)) for _, L, e, *_ in _shells(b)]
        flops = sum(n1 * n2 * (45 + 6 * _nherm(a + c)) for i, (a, n1) in enumerate(prims) for c, n2 in prims[:i + 1])
        m = case["charges"] + b.mol.natom
        return {"bytes": 24.0 * b.nbasis ** 2 + 32.0 * m, "flops": float(flops) * m}
    by, fl = _fock_work(b, case["cut"])
    if kind == "scf":   # about eleven cycles: the builds and some forty multiplications of n x n matrices each
        return {"bytes": 11 * by, "flops": 11 * (fl + 40 * 2.0 * b.nbasis ** 3)}
    if case["delta"]:   # a smaller density moves the screen
        by, fl = _fock_work(b, min(1e-4, case["cut"] / case["delta"]))
    return {"bytes": by * (2 if kind == "uhf" else 1), "flops": fl * (1.5 if kind == "uhf" else 1.0)}


# ---------------------------------------------------------------- 64-bit values from the definitions
def _boys(M, T):
    """[F_0 .. F_M](T): the convergent series and downward recursion to T = 30, erf and upward recursion above."""
    small = torch.clamp(T, max=30.0)
    term = torch.full_like(T, 1.0 / (2 * M + 1))
    total = term.clone()
    for k in range(1, 140):
        term = term * (2.0 * small / (2 * M + 2 * k + 1))
        total += term
    e = torch.exp(-small)
    lo = [None] * (M + 1)
    lo[M] = e * total
    for m in range(M, 0, -1):
        lo[m - 1] = (2.0 * small * lo[m] + e) / (2 * m - 1)
    big = torch.clamp(T, min=30.0)
    hi = [0.5 * torch.sqrt(math.pi / big) * torch.erf(torch.sqrt(big))]
    e = torch.exp(-big)
    for m in range(M):
        hi.append(((2 * m + 1) * hi[m] - e) / (2.0 * big))
    return [torch.where(T <= 30.0, a, c) for a, c in zip(lo, hi)]


def _tuv(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _hermite_coulomb(L, alpha, X, Y, Z):
    """{(t, u, v): R_tuv} for t + u + v <= L (McMurchie-Davidson), over arrays of any shape."""
    F = _boys(L, alpha * (X * X + Y * Y + Z * Z))
    level = {}
    for m in range(L, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** m * F[m]}
        for t, u, v in sorted(_tuv(L - m), key=sum)[1:]:
            if t:
                r = X * level[(t - 1, u, v)] + ((t - 1) * level[(t - 2, u, v)] if t > 1 else 0.0)
            elif u:
                r = Y * level[(t, u - 1, v)] + ((u - 1) * level[(t, u - 2, v)] if u > 1 else 0.0)
            else:
                r = Z * level[(t, u, v - 1)] + ((v - 1) * level[(t, u, v - 2)] if v > 1 else 0.0)
            new[(t, u, v)] = r
        level = new
    return level


def _hermite_1d(i, j, a, b, xab):
    """E_t^{ij}, t = 0 .. i + j, of two 1-d Gaussians (without the exponential prefactor) at distance xab."""
    p = a + b
    pa, pb = -b / p * xab, a / p * xab
    E = {(0, 0): [1.0]}
    for ii in range(i + 1):
        for jj in range(j + 1):
            if (ii, jj) == (0, 0):
                continue
            low, s = (E[(ii - 1, jj)], pa) if ii else (E[(ii, jj - 1)], pb)
            g = lambda t: low[t] if 0 <= t < len(low) else 0.0  # noqa: E731
            E[(ii, jj)] = [g(t - 1) / (2 * p) + s * g(t) + (t + 1) * g(t + 1) for t in range(ii + jj + 1)]
    return E[(i, j)]


def _pair_classes(shells, dev):
    """Per (La, Lb): primitive pairs' exponents, centres, pair numbers and Hermite coefficients [prims, na nb, tuv]
    (contraction coefficients, factors and the Gaussian prefactor inside), and every pair's first functions."""
    cls = {}
    for i, A in enumerate(shells):
        for B in shells[:i + 1]:
            cls.setdefault((A[1], B[1]), []).append((A, B))
    out = []
    for (La, Lb), pairs in cls.items():
        tuv = _tuv(La + Lb)
        at = {x: k for k, x in enumerate(tuv)}
        p, P, num, E = [], [], [], []
        for k, (A, B) in enumerate(pairs):
            ab = A[0] - B[0]
            for ea, ca in zip(A[2], A[3]):
                for eb, cb in zip(B[2], B[3]):
                    s = ea + eb
                    pre = ca * cb * math.exp(-ea * eb / s * float(ab @ ab))
                    p.append(s)
                    P.append((ea * A[0] + eb * B[0]) / s)
                    num.append(k)
                    one = [{(x, y): _hermite_1d(x, y, ea, eb, ab[d]) for x in range(La + 1) for y in range(Lb + 1)}
                           for d in range(3)]
                    M = np.zeros((len(A[6]) * len(B[6]), len(tuv)))
                    for x, (fa, na) in enumerate(zip(A[6], A[5])):
                        for y, (fb, nb) in enumerate(zip(B[6], B[5])):
                            Ex, Ey, Ez = (one[d][(fa[d], fb[d])] for d in range(3))
                            for t, vt in enumerate(Ex):
                                for u, vu in enumerate(Ey):
                                    for v, vv in enumerate(Ez):
                                        M[x * len(B[6]) + y, at[(t, u, v)]] = pre * na * nb * vt * vu * vv
                    E.append(M)
        ten = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device=dev)  # noqa: E731
        out.append({"L": La + Lb, "tuv": tuv, "p": ten(p), "P": ten(P), "E": ten(E), "npair": len(pairs),
                    "num": torch.tensor(num, device=dev), "na": len(pairs[0][0][6]), "nb": len(pairs[0][1][6]),
                    "fa": torch.tensor([A[4] for A, _ in pairs], device=dev),
                    "fb": torch.tensor([B[4] for _, B in pairs], device=dev)})
    return out


def _eri(shells, n, dev):
    """The whole tensor (ij|kl), n^4 values."""
    G = torch.zeros((n, n, n, n), dtype=torch.float64, device=dev)
    cl = _pair_classes(shells, dev)

    def functions(c):
        a = c["fa"][:, None] + torch.arange(c["na"], device=dev)
        b = c["fb"][:, None] + torch.arange(c["nb"], device=dev)
        return a[:, :, None].expand(-1, -1, c["nb"]).reshape(-1), b[:, None, :].expand(-1, c["na"], -1).reshape(-1)

    for bra in cl:
        for ket in cl:
            L, tb, tk = bra["L"] + ket["L"], bra["tuv"], ket["tuv"]
            nab, ncd = bra["na"] * bra["nb"], ket["na"] * ket["nb"]
            V = torch.zeros((bra["npair"], nab, ket["npair"], ncd), dtype=torch.float64, device=dev)
            sign = torch.tensor([(-1.0) ** sum(x) for x in tk], dtype=torch.float64, device=dev)
            Ek = (ket["E"] * sign).transpose(1, 2).contiguous()
            nk = len(ket["p"])
            step = max(1, int(2e8 / (nk * (len(tb) * max(len(tk), ncd) + 4 * _nherm(L)))))
            for i in range(0, len(bra["p"]), step):
                p, P = bra["p"][i:i + step, None], bra["P"][i:i + step]
                q, Q = ket["p"][None], ket["P"]
                d = P[:, None, :] - Q[None]
                R = _hermite_coulomb(L, p * q / (p + q), d[..., 0], d[..., 1], d[..., 2])
                pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
                part = torch.zeros((len(P), len(tb), ket["npair"], ncd), dtype=torch.float64, device=dev)
                for k, (t, u, v) in enumerate(tb):
                    rows = torch.stack([R[(t + a, u + b, v + c)] for a, b, c in tk], dim=-1) * pre[..., None]
                    part[:, k].index_add_(1, ket["num"], torch.einsum("bkt,ktc->bkc", rows, Ek))
                V.index_add_(0, bra["num"][i:i + step], torch.einsum("bat,btkc->bakc", bra["E"][i:i + step], part))
            a, b = functions(bra)
            c, d = functions(ket)
            W = V.reshape(len(a), len(c))
            for x, y in ((a, b), (b, a)):
                for z, w in ((c, d), (d, c)):
                    G[x[:, None], y[:, None], z[None], w[None]] = W
    return G


def _one_electron(b, ext, dev):
    """S, T and V (nuclei and external charges) from the one-electron form of the basis."""
    n = b.nbasis
    shells, f = [], 0
    while f < n:   # components of a shell follow one another
        L = int(b.itype[:, f].sum())
        m, k = (L + 1) * (L + 2) // 2, int(b.ncontract[f])
        comps = [tuple(int(x) for x in b.itype[:, g]) for g in range(f, f + m)]
        ratio = b.dcoeff[0, f:f + m] / b.dcoeff[0, f]
        shells.append((b.xyz[int(b.ncenter[f]) - 1], L, b.aexp[:k, f], b.dcoeff[:k, f], f, ratio, comps))
        f += m
    S, T, V = (torch.zeros((n, n), dtype=torch.float64, device=dev) for _ in range(3))
    xyz = np.concatenate([b.xyz, ext[0]]) if ext is not None else b.xyz
    q = np.concatenate([b.mol.Z.astype(float), ext[1]]) if ext is not None else b.mol.Z.astype(float)
    xyz, q = (torch.tensor(v, dtype=torch.float64, device=dev) for v in (xyz, q))
    for c in _pair_classes(shells, dev):
        step = max(1, int(1e8 / (len(q) * 4 * _nherm(c["L"]))))
        out = torch.zeros((c["npair"], c["na"] * c["nb"]), dtype=torch.float64, device=dev)
        for i in range(0, len(c["p"]), step):
            p, d = c["p"][i:i + step], c["P"][i:i + step, None] - xyz[None]
            R = _hermite_coulomb(c["L"], p[:, None], d[..., 0], d[..., 1], d[..., 2])
            r = torch.stack([(R[x] * q).sum(1) for x in c["tuv"]], dim=-1) * (-2.0 * math.pi / p)[:, None]
            out.index_add_(0, c["num"][i:i + step], torch.einsum("bat,bt->ba", c["E"][i:i + step], r))
        a = (c["fa"][:, None, None] + torch.arange(c["na"], device=dev)[:, None]).expand(-1, -1, c["nb"]).reshape(-1)
        w = (c["fb"][:, None, None] + torch.arange(c["nb"], device=dev)[None]).expand(-1, c["na"], -1).reshape(-1)
        V[a, w] = out.reshape(-1)
        V[w, a] = out.reshape(-1)
    Sn, Tn = np.zeros((n, n)), np.zeros((n, n))
    for i, A in enumerate(shells):
        for B in shells[:i + 1]:
            ab = A[0] - B[0]
            for ea, ca in zip(A[2], A[3]):
                for eb, cb in zip(B[2], B[3]):
                    s = ea + eb
                    pre = ca * cb * math.exp(-ea * eb / s * float(ab @ ab)) * (math.pi / s) ** 1.5
                    if abs(pre) < 1e-25:
                        continue
                    o = [{(x, y): _hermite_1d(x, y, ea, eb, ab[k])[0] for x in range(A[1] + 1)
                          for y in range(B[1] + 3)} for k in range(3)]
                    kin = [{(x, y): eb * (2 * y + 1) * o[k][(x, y)] - 2 * eb * eb * o[k][(x, y + 2)]
                            - (0.5 * y * (y - 1) * o[k][(x, y - 2)] if y > 1 else 0.0)
                            for x in range(A[1] + 1) for y in range(B[1] + 1)} for k in range(3)]
                    for x, (fa, na) in enumerate(zip(A[6], A[5])):
                        for y, (fb, nb) in enumerate(zip(B[6], B[5])):
                            s3 = [o[k][(fa[k], fb[k])] for k in range(3)]
                            t3 = [kin[k][(fa[k], fb[k])] for k in range(3)]
                            Sn[A[4] + x, B[4] + y] += pre * na * nb * s3[0] * s3[1] * s3[2]
                            Tn[A[4] + x, B[4] + y] += pre * na * nb * (
                                t3[0] * s3[1] * s3[2] + s3[0] * t3[1] * s3[2] + s3[0] * s3[1] * t3[2])
    low = np.tril(np.ones((n, n), dtype=bool))
    Sn, Tn = (np.where(low, x, x.T) for x in (Sn, Tn))
    return Sn, Tn, V.cpu().numpy()


def _jk(G, D):
    return torch.einsum("ijkl,kl->ij", G, D), torch.einsum("ikjl,kl->ij", G, D)


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kind = case["kind"]
    with torch.no_grad():
        if kind == "scf":
            return None   # a solve stops at its own threshold, not at the fixed point
        if kind == "oei":
            b = _basis(case, seed)
            return _one_electron(b, _charges(case, b, seed), dev) if b.nbasis <= 160 else None
        if kind == "batch":
            st = prepare(case, seed)
            return [_closed(e.basis, D, dev) if e.basis.nbasis <= 60 else None
                    for e, D in zip(st["engines"], st["D"])]
        b = _basis(case, seed)
        if b.nbasis > 200:
            return None
        st = prepare(dict(case, tune=False), seed)
        if kind == "uhf":
            Da, Db = st["Da"].to(dev), st["Db"].to(dev)
            G = _eri(_shells(b), b.nbasis, dev)
            (Ja, Ka), (Jb, Kb) = _jk(G, Da), _jk(G, Db)
            return Ja + Jb - Ka, Ja + Jb - Kb
        got = _closed(b, torch.as_tensor(st["D"]).to(dev), dev)
        return got.cpu().numpy() if kind == "host" else got


def _closed(b, D, dev):
    J, K = _jk(_eri(_shells(b), b.nbasis, dev), D.to(dev))
    return J - 0.5 * K
