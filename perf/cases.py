"""Performance cases of the direct Fock build: what a user's program has this
library do, through its public entry points.

Every case is a plain dict.  ``kind`` says which call it stands for:

* ``scf``       one J/K build of a closed-shell real density, on device matrices
                (``GTODirectTPIContraction.twoBodyContract``) or on host ones
                (``FockBuilder.formRawGD`` into the caller's J, K and G)
* ``complex``   J/K of a complex Hermitian density (a real-time propagation step)
* ``batch``     J/K of many increment densities in one captured CUDA graph
                (``ContractionGraph``)
* ``geometry``  a new geometry: pair and Schwarz set-up (``DirectTPI``) and the
                first J/K build on it
* ``gradient``  J/K contractions of all first derivatives of the integrals
                (``DirectGradContraction.gradTwoBodyContract``)
* ``dirac``     a four-component build (``FourCompFock.formGD``): bare Coulomb,
                LLSS and SSSS, optionally Gaunt, of an uncontracted atom or of
                contracted water molecules

Molecules are seeded water clusters (or one atom); densities come from the
seed.  ``exact`` computes the same matrices with numpy from a full table of
integrals (McMurchie-Davidson over Hermite expansions), for the molecules that
are small enough for it.
"""
import math

import numpy as np
import torch

from chronusq_public_b200 import workloads
from chronusq_public_b200.basis import BasisSet, Molecule
from chronusq_public_b200.contraction import (COULOMB, EXCHANGE, ContractionGraph,
                                              DirectGradContraction, DirectTPI,
                                              GTODirectTPIContraction, TwoBodyContraction)
from chronusq_public_b200.fockbuilder import FockBuilder, FourCompFock

CUTOFF = 1e-2          # FP32 cutoff of the mixed-precision builds (the bench's default)
EXACT_FUNCTIONS = 30   # largest basis whose full integral table takes seconds in numpy


def listed():
    return [
        # the smallest call there is in an SCF loop: one water molecule
        dict(name="water", kind="scf", waters=1, basis="cc-pvdz", precision="fp64",
             where="device"),
        # the benchmark's build end to end: host matrices in, J, K and G out
        dict(name="water16_host_mixed", kind="scf", waters=16, basis="def2-svp",
             precision="mixed", where="host"),
        # the same molecule in double precision on device matrices
        dict(name="water16", kind="scf", waters=16, basis="def2-svp", precision="fp64",
             where="device"),
        # the largest cluster of the serving stream
        dict(name="water32_mixed", kind="scf", waters=32, basis="cc-pvdz", precision="mixed",
             where="device"),
        # a triple-zeta basis: f shells
        dict(name="water3_f", kind="scf", waters=3, basis="cc-pvtz", precision="fp64",
             where="device"),
        # one step of a real-time propagation
        dict(name="water8_complex", kind="complex", waters=8, basis="cc-pvdz"),
        # 64 increment densities per graph launch
        dict(name="water8_batch64", kind="batch", waters=8, basis="cc-pvdz", densities=64),
        # one step of a geometry optimisation, and every new request of a server
        dict(name="water8_geometry", kind="geometry", waters=8, basis="def2-svp"),
        # the two-electron gradient of the same optimisation
        dict(name="water4_gradient", kind="gradient", waters=4, basis="cc-pvdz"),
        # four-component Dirac-Coulomb build of a heavy atom, uncontracted with f shells
        dict(name="ag_dirac", kind="dirac", atom="Ag", basis="sapporo-dkh3-dzp-2012_no",
             waters=0, precision="fp64", gaunt=False),
        # a small contracted Dirac-Coulomb build with mixed precision
        dict(name="water_dirac_mixed", kind="dirac", atom="", basis="6-31gd", waters=1,
             precision="mixed", gaunt=False),
        # Dirac-Coulomb-Gaunt
        dict(name="water_gaunt", kind="dirac", atom="", basis="6-31gd", waters=1,
             precision="fp64", gaunt=True),
    ]


def _spread(rng, lo, hi):
    """A whole number of lo..hi, evenly over its logarithm."""
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["scf", "scf", "scf", "complex", "batch", "geometry", "gradient",
                       "dirac", "dirac"])
    svp = ["3-21g", "6-31gd", "cc-pvdz", "def2-svp"]
    if kind == "scf":
        basis = rng.choice(svp + ["cc-pvtz"])
        return dict(kind=kind, waters=_spread(rng, 1, 4 if basis == "cc-pvtz" else 31),
                    basis=basis, precision=rng.choice(["fp64", "mixed"]),
                    where=rng.choice(["device", "host"]))
    if kind == "complex":
        return dict(kind=kind, waters=_spread(rng, 1, 12), basis=rng.choice(svp))
    if kind == "batch":
        return dict(kind=kind, waters=_spread(rng, 1, 8), basis=rng.choice(svp),
                    densities=_spread(rng, 2, 64))
    if kind == "geometry":
        return dict(kind=kind, waters=_spread(rng, 1, 16), basis=rng.choice(svp))
    if kind == "gradient":
        return dict(kind=kind, waters=_spread(rng, 1, 4), basis=rng.choice(svp))
    if rng.random() < 0.5:
        return dict(kind=kind, atom=rng.choice(["Ni", "Cu", "Zn", "Br", "Kr", "Mo", "Pd"]),
                    basis="sapporo-dkh3-dzp-2012_no", waters=0,
                    precision=rng.choice(["fp64", "mixed"]), gaunt=False)
    return dict(kind=kind, atom="", basis=rng.choice(["3-21g", "6-31gd", "cc-pvdz"]),
                waters=rng.choice([1, 1, 2]),
                precision=rng.choice(["fp64", "mixed"]), gaunt=rng.random() < 0.4)


# ------------------------------------------------------------------ inputs
def _molecule(case, seed=0):
    if case["waters"] == 0:
        return Molecule.from_angstrom([(case["atom"], 0.0, 0.0, 0.0)])
    n = case["waters"]
    # the serving stream's density of molecules
    return workloads.water_cluster(n, seed=40 + n + 1000 * seed,
                                   box=max(6.0, 10.0 * (n / 16.0) ** (1 / 3)))


def _basis(case, seed=0):
    return BasisSet.build(_molecule(case, seed), case["basis"],
                          uncontract=case["waters"] == 0)


def _occupied(case):
    return 5 * case["waters"]


def _density(case, S, T, seed):
    """The host densities of a case: one matrix, a list of them, or the four
    Pauli components."""
    kind, N = case["kind"], S.shape[0]
    if kind in ("scf", "geometry", "gradient"):
        return workloads.occupied_density(S, _occupied(case), seed)
    if kind == "complex":
        rng = np.random.default_rng(seed)
        C = rng.normal(size=(N, _occupied(case))) + 1j * rng.normal(size=(N, _occupied(case)))
        w, V = np.linalg.eigh(C.conj().T @ S @ C)
        C = C @ (V @ np.diag(w ** -0.5) @ V.conj().T)
        return C @ C.conj().T
    if kind == "batch":
        return workloads.delta_densities(N, case["densities"], seed_base=1000 * (seed + 1))
    nocc = 47 if case["waters"] == 0 else 2 * _occupied(case)
    return workloads.spinor_density_4c(S, T, nocc, seed)


def _cuda(a):
    """A column-major CUDA copy of a host matrix."""
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().T


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    # a geometry step's molecule changes with the seed, the others' stays
    basis = _basis(case, seed % 1000 if kind == "geometry" else 0)
    tpi = DirectTPI(basis)
    S, T = tpi.one_electron()
    D = _density(case, S, T, seed)
    N = basis.nbasis
    s.update(basis=basis, tpi=tpi)
    if kind == "geometry":
        tpi.close()
        s["tpi"] = None
    if kind == "scf" and case["where"] == "host":
        s.update(D=D, fock=FockBuilder(tpi),
                 out=[np.zeros((N, N), order="F") for _ in range(3)])
    elif kind == "dirac":
        s.update(D=[_cuda(d) for d in D],
                 fock=FourCompFock(tpi, Gaunt=case["gaunt"]))
    elif kind == "batch":
        X = [_cuda(d) for d in D]
        out = torch.zeros((len(X), 2, N, N), dtype=torch.float64, device="cuda")
        lst = []
        for i, x in enumerate(X):
            lst.append(TwoBodyContraction(x, out[i, 0].T, True, COULOMB))
            lst.append(TwoBodyContraction(x, out[i, 1].T, True, EXCHANGE))
        s.update(out=out, graph=ContractionGraph(tpi, lst))
    elif kind == "gradient":
        natom = 3 * case["waters"]
        X = _cuda(D)
        out = torch.zeros((3 * natom, 2, N, N), dtype=torch.float64, device="cuda")
        s.update(out=out, grad=DirectGradContraction(tpi),
                 atoms=np.array([sh.atom for sh in basis.shells], dtype=np.int32),
                 lists=[[TwoBodyContraction(X, out[g, 0].T, True, COULOMB),
                         TwoBodyContraction(X, out[g, 1].T, True, EXCHANGE)]
                        for g in range(3 * natom)])
    else:
        X = _cuda(D)
        out = torch.zeros((2, N, N), dtype=X.dtype, device="cuda")
        s.update(out=out, lists=[TwoBodyContraction(X, out[0].T, True, COULOMB),
                                 TwoBodyContraction(X, out[1].T, True, EXCHANGE)])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "scf" and case["where"] == "host":
        J, K, G = s["out"]
        s["fock"].formRawGD(s["D"], precision=case["precision"], fp32_cutoff=CUTOFF,
                            J=J, K=K, G=G)
        return [J, K, G]
    if kind == "dirac":
        return s["fock"].formGD(s["D"], precision=case["precision"], fp32_cutoff=CUTOFF,
                                stream=_stream())
    s["out"].zero_()
    if kind == "batch":
        s["graph"].launch(stream=_stream())
    elif kind == "gradient":
        s["grad"].gradTwoBodyContract(s["lists"], s["atoms"], stream=_stream())
    elif kind == "geometry":
        tpi = DirectTPI(s["basis"])
        GTODirectTPIContraction(tpi).twoBodyContract(s["lists"], stream=_stream())
        tpi.close()
    else:
        GTODirectTPIContraction(s["tpi"]).twoBodyContract(
            s["lists"], precision=case.get("precision", "fp64"), fp32_cutoff=CUTOFF,
            stream=_stream())
    return s["out"]


# ---------------------------------------------------- work and tolerances
def _pair_counts(basis):
    """{(la, lb, bin): [shell pairs, primitive pairs, functions]} of the pairs of shells,
    binned by the whole decades of their overlap exp(-mu R^2)."""
    sh = basis.shells
    O = np.array([s.origin for s in sh])
    out = {}
    for i in range(len(sh)):
        for j in range(i + 1):
            R2 = float(((O[i] - O[j]) ** 2).sum())
            a, b = np.asarray(sh[i].alpha)[:, None], np.asarray(sh[j].alpha)[None, :]
            e = (a * b / (a + b)) * R2 / math.log(10.0)
            k = int(e.min())
            if k > 12:
                continue
            la, lb = max(sh[i].l, sh[j].l), min(sh[i].l, sh[j].l)
            c = out.setdefault((la, lb, k), [0, 0, 0])
            c[0] += 1
            c[1] += int((e <= 12.0).sum())
            c[2] += sh[i].size * sh[j].size
    return out


def _herm(n):
    return (n + 1) * (n + 2) * (n + 3) // 6


def _cart(l):
    return (l + 1) * (l + 2) // 2


def _quartet_flops(la, lb, lc, ld, db, dk, ob, ok):
    """Operations of one primitive quartet: the Hermite recursion of order
    la + lb + lc + ld + db + dk, then the two expansions, with ob and ok
    operator components of the differentiated bra and ket."""
    lab, lcd = la + lb + db, lc + ld + dk
    nab, ncd = _cart(la) * _cart(lb) * ob, _cart(lc) * _cart(ld) * ok
    hab, hcd = _herm(lab), _herm(lcd)
    R = 3 * sum(_herm(lab + lcd - n) for n in range(lab + lcd + 1))
    return 20 + R + 2 * hab * min(hcd * ncd + ncd * nab, hcd * nab + ncd * nab)


def work(case):
    """Each matrix read or written once, and the McMurchie-Davidson operations
    of the unique primitive quartets whose overlaps' product reaches 1e-11."""
    basis = _basis(case)
    N, kind = basis.nbasis, case["kind"]
    counts = list(_pair_counts(basis).items())
    # (bra order raised, ket order raised, bra components, ket components, weight)
    terms = {"gradient": [(1, 1, 3, 1, 3.0)],
             "dirac": [(0, 0, 1, 1, 1.0), (2, 0, 4, 1, 2.0), (2, 2, 4, 4, 1.0)]}.get(
                 kind, [(0, 0, 1, 1, 1.0)])
    if case.get("gaunt"):
        terms = terms + [(1, 1, 3, 3, 4.0)]
    updates = {"complex": 18, "batch": 12 * case.get("densities", 1), "gradient": 12 * 9,
               "dirac": 36 * 16}.get(kind, 12)
    flops = 0.0
    for (la, lb, k), (n1, p1, f1) in counts:
        for (lc, ld, m), (n2, p2, f2) in counts:
            if k + m > 11:
                continue
            for db, dk, ob, ok, w in terms:
                flops += 0.5 * p1 * p2 * w * _quartet_flops(la, lb, lc, ld, db, dk, ob, ok)
            flops += 0.5 * f1 * f2 * updates
    matrices = {"complex": 6, "batch": 3 * case.get("densities", 1),
                "gradient": 1 + 18 * case["waters"], "dirac": 2 * 4 * 4 * 2}.get(kind, 3)
    if case.get("where") == "host":
        matrices += 1
    return dict(bytes=8.0 * matrices * N * N, flops=flops)


def tolerance(case):
    """Double precision: the screening threshold (1e-12 per quartet) and sums
    in another order; mixed: quartets of bound below 1e-2 in FP32."""
    if case.get("precision") == "mixed":
        return dict(rel=1e-7, max=1e-5)
    return dict(rel=1e-10, max=1e-8)


# ------------------------------------------------------------------- exact
def _boys(L, T):
    """F_0..F_L (L + 1, n): the convergent series and the downward recursion
    below T = 40, the asymptotic F_0 and the upward recursion above it."""
    F = np.zeros((L + 1, T.size))
    lo = T < 40.0
    t = T[lo]
    if t.size:
        term = np.full(t.size, 1.0 / (2 * L + 1))
        s = term.copy()
        for k in range(1, 400):
            term = term * (2.0 * t / (2 * L + 2 * k + 1))
            s += term
            if (term <= 1e-17 * s).all():
                break
        e = np.exp(-t)
        f = e * s
        F[L, lo] = f
        for m in range(L - 1, -1, -1):
            f = (2.0 * t * f + e) / (2 * m + 1)
            F[m, lo] = f
    t = T[~lo]
    if t.size:
        f, e = 0.5 * np.sqrt(np.pi / t), np.exp(-t)
        F[0, ~lo] = f
        for m in range(L):
            f = ((2 * m + 1) * f - e) / (2.0 * t)
            F[m + 1, ~lo] = f
    return F


def _hermites(L):
    return [(t, u, n - t - u) for n in range(L + 1) for t in range(n, -1, -1)
            for u in range(n - t, -1, -1)]


def _hermite_integrals(L, alpha, XYZ):
    """R_tuv for t + u + v <= L: {(t, u, v): (n,)}."""
    F = _boys(L, alpha * (XYZ ** 2).sum(0))
    cur = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** n * F[n]}
        for h in _hermites(L - n)[1:]:
            x = next(k for k in range(3) if h[k])
            lower = list(h)
            lower[x] -= 1
            v = XYZ[x] * cur[tuple(lower)]
            if lower[x]:
                low2 = list(lower)
                low2[x] -= 1
                v = v + lower[x] * cur[tuple(low2)]
            new[h] = v
        cur = new
    return cur


def _hermite_1d(i, j, p, pa, pb):
    """E^{ij}_t, t = 0..i+j, of x_A^i x_B^j exp(-p x_P^2) in Hermite Gaussians."""
    if i == 0 and j == 0:
        return np.ones(1)
    e = _hermite_1d(i - 1, j, p, pa, pb) if i else _hermite_1d(i, j - 1, p, pa, pb)
    out = np.zeros(i + j + 1)
    out[:-1] += (pa if i else pb) * e
    out[1:] += e / (2.0 * p)
    out[:-2] += np.arange(1, e.size) * e[1:]
    return out


def _derivative(i, a, on):
    """(factor, power) terms of d^on/dx^on x^i exp(-a x^2), on = 0 or 1."""
    if not on:
        return [(1.0, i)]
    return [(-2.0 * a, i + 1)] + ([(float(i), i - 1)] if i else [])


# operator components of a pair density: sums of (factor, axis of the
# derivative on the first function or None, on the second or None)
_PLAIN = [[(1.0, None, None)]]
_FIRST = [[(1.0, x, None)] for x in range(3)]
_SECOND = [[(1.0, None, x)] for x in range(3)]
_SPIN = [[(1.0, x, x) for x in range(3)]] + [
    [(1.0, (x + 1) % 3, (x + 2) % 3), (-1.0, (x + 2) % 3, (x + 1) % 3)] for x in range(3)]


def _pair_densities(basis, ops):
    """Hermite expansions of every (operator, function, function) pair density,
    by primitive pair: {order: [(P, p, shell pair, (ops, na, nb, H) array)]}."""
    rise = max((f is not None) + (s is not None) for op in ops for _, f, s in op)
    T = [_spherical(s) for s in basis.shells]
    out = {}
    for i1, A in enumerate(basis.shells):
        for i2, B in enumerate(basis.shells):
            L = A.l + B.l + rise
            where = {h: k for k, h in enumerate(_hermites(L))}
            ca, cb = _components(A.l), _components(B.l)
            for a, wa in zip(A.alpha, A.coef):
                for b, wb in zip(B.alpha, B.coef):
                    p = a + b
                    P = (a * A.origin + b * B.origin) / p
                    w = wa * wb * math.exp(-a * b / p * ((A.origin - B.origin) ** 2).sum())
                    E = {}

                    def axis(x, i, j, da, db):
                        key = (x, i, j, da, db)
                        if key not in E:
                            v = np.zeros(L + 1)
                            for f, ii in _derivative(i, a, da):
                                for g, jj in _derivative(j, b, db):
                                    e = _hermite_1d(ii, jj, p, P[x] - A.origin[x],
                                                    P[x] - B.origin[x])
                                    v[:e.size] += f * g * e
                            E[key] = v
                        return E[key]

                    C = np.zeros((len(ops), len(ca), len(cb), len(where)))
                    for o, op in enumerate(ops):
                        for f, d1, d2 in op:
                            for m, u in enumerate(ca):
                                for n, v in enumerate(cb):
                                    e = [axis(x, u[x], v[x], d1 == x, d2 == x)
                                         for x in range(3)]
                                    C[o, m, n] += f * w * np.array(
                                        [e[0][t] * e[1][y] * e[2][z] for t, y, z in where])
                    C = np.einsum("omnh,mi,nj->oijh", C, T[i1], T[i2])
                    out.setdefault((L, C.shape[1], C.shape[2]), []).append((P, p, (i1, i2), C))
    return out


def _components(l):
    return [(l - a, a - b, b) for a in range(l + 1) for b in range(a + 1)]


def _spherical(shell):
    """Cartesian components to the shell's functions: real solid harmonics
    r^l Y_lm from their recursion in l, scaled as the Cartesian x^l is."""
    l = shell.l
    if not shell.pure:
        return np.eye(_cart(l))
    # polynomials {(i, j, k): c}; the complex harmonic of m is (x + iy)^m
    # times Pi_l^m(z, r^2), with Pi from (l - m) Pi_l = (2l - 1) z Pi_(l-1) -
    # (l + m - 1) r^2 Pi_(l-2)
    def times(p, q):
        r = {}
        for a, u in p.items():
            for b, v in q.items():
                k = (a[0] + b[0], a[1] + b[1], a[2] + b[2])
                r[k] = r.get(k, 0) + u * v
        return r

    x_iy, z = {(1, 0, 0): 1.0, (0, 1, 0): 1j}, {(0, 0, 1): 1.0}
    r2 = {(2, 0, 0): 1.0, (0, 2, 0): 1.0, (0, 0, 2): 1.0}
    T = np.zeros((_cart(l), 2 * l + 1))
    comps = _components(l)
    for m in range(l + 1):
        dfact = 1.0
        for k in range(1, 2 * m, 2):
            dfact *= k
        prev, cur = {}, {(0, 0, 0): dfact}
        for k in range(m + 1, l + 1):
            nxt = {q: (2 * k - 1) * v / (k - m) for q, v in times(z, cur).items()}
            for q, v in times(r2, prev).items():
                nxt[q] = nxt.get(q, 0) - (k + m - 1) * v / (k - m)
            prev, cur = cur, nxt
        for _ in range(m):
            cur = times(cur, x_iy)
        norm = math.sqrt((2.0 if m else 1.0) * math.factorial(l - m) / math.factorial(l + m))
        for q, v in cur.items():
            T[comps.index(q), l + m] = norm * np.real(v)
            if m:
                T[comps.index(q), l - m] = norm * np.imag(v)
    return T


def _integrals(basis, bra, ket):
    """(bra operators, N, N, ket operators, N, N) table of (mu nu | la si)."""
    B, K = _pair_densities(basis, bra), _pair_densities(basis, ket)
    N, off, size = basis.nbasis, basis.offsets, basis.sizes
    V = np.zeros((len(bra), N, N, len(ket), N, N))
    for (Lb, na, nb), bl in B.items():
        hb = np.array(_hermites(Lb))
        for (Lk, nc, nd), kl in K.items():
            hk = _hermites(Lk)
            index = {h: n for n, h in enumerate(_hermites(Lb + Lk))}
            gather = np.array([[index[tuple(np.add(u, v))] for v in hk] for u in hb])
            sign = np.array([(-1.0) ** sum(v) for v in hk])
            Q = np.array([k[0] for k in kl]).T
            q = np.array([k[1] for k in kl])
            Ck = np.array([k[3] for k in kl]).reshape(len(kl), -1, len(hk)) * sign[None, None]
            kets = {}
            for n, k in enumerate(kl):
                kets.setdefault(k[2], []).append(n)
            step = max(1, int(1.5e7 // (len(kl) * max(gather.size, len(index)))))
            for i0 in range(0, len(bl), step):
                part = bl[i0:i0 + step]
                P = np.array([b[0] for b in part]).T
                p = np.array([b[1] for b in part])[:, None]
                alpha = (p * q / (p + q)).ravel()
                pref = (2.0 * math.pi ** 2.5 / (p * q * np.sqrt(p + q))).ravel()
                R = _hermite_integrals(Lb + Lk, alpha,
                                       (P[:, :, None] - Q[:, None, :]).reshape(3, -1))
                R = np.stack([R[h] * pref for h in index]).reshape(
                    len(index), len(part), len(kl))
                for n, b in enumerate(part):
                    Cb = b[3].reshape(-1, len(hb))
                    W = np.einsum("ch,hkj->jck", Cb, R[gather, n], optimize=True)
                    W = np.matmul(W, Ck.transpose(0, 2, 1))
                    a1, a2 = b[2]
                    for (c1, c2), js in kets.items():
                        blk = W[js].sum(0).reshape(len(bra), na, nb, len(ket), nc, nd)
                        V[:, off[a1]:off[a1] + size[a1], off[a2]:off[a2] + size[a2], :,
                          off[c1]:off[c1] + size[c1], off[c2]:off[c2] + size[c2]] += blk
    return V


def _spin_blocks(M, N):
    """Pauli components (2N x 2N, large component first) to spin blocks
    {(row, column): [mu, s, nu, s']}."""
    S, X, Y, Z = M
    out = {}
    for r in range(2):
        for c in range(2):
            at = (slice(r * N, (r + 1) * N), slice(c * N, (c + 1) * N))
            b = np.zeros((N, 2, N, 2), dtype=complex)
            b[:, 0, :, 0], b[:, 1, :, 1] = (S[at] + Z[at]) / 2, (S[at] - Z[at]) / 2
            b[:, 0, :, 1], b[:, 1, :, 0] = (X[at] - 1j * Y[at]) / 2, (X[at] + 1j * Y[at]) / 2
            out[r, c] = b
    return out


def _pauli(blocks, N):
    G = [np.zeros((2 * N, 2 * N), dtype=complex) for _ in range(4)]
    for (r, c), b in blocks.items():
        at = (slice(r * N, (r + 1) * N), slice(c * N, (c + 1) * N))
        aa, bb, ab, ba = b[:, 0, :, 0], b[:, 1, :, 1], b[:, 0, :, 1], b[:, 1, :, 0]
        for g, m in zip(G, (aa + bb, ab + ba, 1j * (ab - ba), aa - bb)):
            g[at] += m
    return G


_SIGMA = np.array([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]], dtype=complex)


def _dirac_coulomb(basis, D):
    """J - K over kinetically balanced spinors: chi, and sigma.p chi / 2c, whose
    pair densities are (dot + i sigma . cross) of the gradients / 4c^2."""
    N, c2 = basis.nbasis, 1.0 / (4.0 * workloads.SPEED_OF_LIGHT ** 2)
    spin = [np.eye(2, dtype=complex)[None],
            c2 * np.concatenate([np.eye(2, dtype=complex)[None], 1j * _SIGMA])]
    ops = [_PLAIN, _SPIN]
    ss = _integrals(basis, _SPIN, _SPIN)
    ls = _integrals(basis, _PLAIN, _SPIN)
    V = {(0, 0): _integrals(basis, _PLAIN, _PLAIN), (0, 1): ls,
         (1, 0): ls.transpose(3, 4, 5, 0, 1, 2), (1, 1): ss}
    Db = _spin_blocks(D, N)
    G = {}
    for x in range(2):
        pot = np.zeros((len(ops[x]), N, N), dtype=complex)
        for y in range(2):
            rho = np.einsum("otu,duct->ocd", spin[y], Db[y, y])
            pot += np.einsum("oabpcd,pcd->oab", V[x, y], rho)
        G[x, x] = np.einsum("ost,oab->asbt", spin[x], pot)
    for x in range(2):
        for y in range(2):
            # (P S | R Q) D_SR with P, S of type x and R, Q of type y
            W = np.einsum("ost,pum,ctdu->opscdm", spin[x], spin[y], Db[x, y], optimize=True)
            K = np.einsum("oacpdb,opscdm->asbm", V[x, y], W, optimize=True)
            G[x, y] = G.get((x, y), 0) - K
    return _pauli(G, N)


def _gaunt(basis, D):
    """J - K of -alpha_1 . alpha_2 / r12: the pair densities of mixed type are
    (-i / 2c) sigma_k sigma_j chi d_j chi' and its conjugate."""
    N, c2 = basis.nbasis, 1.0 / (4.0 * workloads.SPEED_OF_LIGHT ** 2)
    T = _integrals(basis, _SECOND, _SECOND).transpose(0, 3, 1, 2, 4, 5)
    pp = np.einsum("iab,jbc->ijac", _SIGMA, _SIGMA)
    ll = c2 * np.einsum("kjab,klcd->jlabcd", pp, pp)
    lr = -c2 * np.einsum("kjab,lkcd->jlabcd", pp, pp)
    rl = -c2 * np.einsum("jkab,klcd->jlabcd", pp, pp)
    Db = _spin_blocks(D, N)

    def two(spec, m, d):
        return np.einsum(spec, m, T, d, optimize=True)

    LL, LS, SL, SS = Db[0, 0], Db[0, 1], Db[1, 0], Db[1, 1]
    ls = (two("jlxytu,jlabcd,duct->axby", ll, SL) + two("jlxytu,jlabcd,cudt->axby", lr, LS)
          - two("jlxuty,jlabcd,buct->axdy", ll, SL))
    G = {(0, 0): -two("jlxuty,jlabcd,budt->axcy", lr, SS),
         (1, 1): -two("jlxuty,jlabcd,auct->bxdy", rl, LL), (0, 1): ls,
         (1, 0): ls.conj().transpose(2, 3, 0, 1)}
    return _pauli(G, N)


def exact(case, seed):
    basis = _basis(case, seed % 1000 if case["kind"] == "geometry" else 0)
    if basis.nbasis > EXACT_FUNCTIONS:
        return None
    tpi = DirectTPI(basis)  # the overlap that the inputs' orbitals are orthonormal in
    S, T = tpi.one_electron()
    tpi.close()
    D = _density(case, S, T, seed)
    kind, N = case["kind"], basis.nbasis
    if kind == "dirac":
        G = _dirac_coulomb(basis, D)
        if case["gaunt"]:
            G = [a + b for a, b in zip(G, _gaunt(basis, D))]
        return G
    if kind == "gradient":
        # d/dR = -d/dr of the functions on the atom, on each of the four places
        A = _integrals(basis, _FIRST, _PLAIN)[:, :, :, 0]
        atom = np.concatenate([np.full(sh.size, sh.atom) for sh in basis.shells])
        out = np.zeros((3 * (int(atom.max()) + 1), 2, N, N))
        for g in range(out.shape[0]):
            B = -A[g % 3] * (atom == g // 3)[:, None, None, None]
            B = B + B.transpose(1, 0, 2, 3)
            B = B + B.transpose(2, 3, 0, 1)
            out[g, 0] = np.einsum("abcd,cd->ab", B, D)
            out[g, 1] = np.einsum("acbd,cd->ab", B, D)
        return out
    V = _integrals(basis, _PLAIN, _PLAIN)[0, :, :, 0]
    flat = V.reshape(N * N, N * N)
    cross = V.transpose(0, 2, 1, 3).reshape(N * N, N * N)

    def jk(d):
        d = np.asarray(d)
        return ((flat @ np.ascontiguousarray(d).reshape(-1).real).reshape(N, N).astype(d.dtype),
                (cross @ np.ascontiguousarray(d).reshape(-1)).reshape(N, N))

    if kind == "batch":
        return np.stack([np.stack([m.T for m in jk(d)]) for d in D])
    J, K = jk(D)
    if kind == "scf" and case["where"] == "host":
        return [J, K, 2.0 * J - K]
    return np.stack([J.T, K.T])  # the rows of `run`'s tensor are columns
