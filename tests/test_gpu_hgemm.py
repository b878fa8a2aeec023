"""The Hermite-matrix engine (csrc/cqf_hgemm.cuh) at the sizes where its work
split changes, against the oracle: contracted f pairs (several chunks of rows
and columns, the integrals made again for each), long contractions (a
quartet's primitives in batches of 32 and over several blocks), one single
shell (tiles almost empty), and FP32 Hermite integrals.  FP64 results agree
to 1e-11 of the largest element (sums of some 1e4 terms in another order);
mixed ones, at a cutoff that divides the quartets, to 1e-6 (FP32 integrals carry
a few 1e-7 of their bounds, which are of the outputs' size here)."""
import numpy as np
import pytest

import oracle as O
from chronusq_public_b200 import _cabi, workloads
from chronusq_public_b200.basis import BasisSet, Molecule, parse_gbs
from chronusq_public_b200.contraction import (COULOMB, EXCHANGE, GAUNT, LLSS, SSSS,
                                              ContractionGraph,
                                              DirectGradContraction, DirectTPI,
                                              GTODirectRelERIContraction,
                                              GTODirectTPIContraction, TwoBodyContraction)
from test_gpu_gaunt import OUTS_C, OUTS_X, gaunt_inputs
from test_gpu_rel import OUTS, max_rel, rel_inputs
from test_zz_no_alloc import _contract as noalloc_contract

pytestmark = pytest.mark.gpu

BASES = {
    # contracted f on two centres, and a pure s partner
    "f2": ("He 0\nF 2 1.00\n  1.7 0.4\n  0.6 0.7\nS 1 1.00\n  0.8 1.0\n",
           "H 0\nF 2 1.00\n  1.1 0.5\n  0.4 0.6\n"),
    # 11 x 11 primitive pairs of s, with a contracted p
    "long": ("He 0\nS 11 1.00\n" + "".join("  %g %g\n" % (0.12 * 2.2 ** k, 0.2 + 0.05 * k)
                                           for k in range(11)) + "P 3 1.00\n  2.9 0.3\n"
             "  0.9 0.6\n  0.3 0.4\n", "H 0\nS 2 1.00\n  1.9 0.3\n  0.4 0.8\n"),
    # f beside an s of 8 primitives (64 x 64 primitive quartets), p, d, f
    "mix": ("He 0\nS 8 1.00\n" + "".join("  %g %g\n" % (0.15 * 2.6 ** k, 0.2 + 0.1 * k)
                                          for k in range(8)) + "F 1 1.00\n  1.3 1.0\n",
            "H 0\nS 2 1.00\n  1.9 0.3\n  0.4 0.8\nP 1 1.00\n  0.7 1.0\nD 1 1.00\n  0.9 1.0\n"
            "F 1 1.00\n  0.8 1.0\n"),
    "one": ("He 0\nS 1 1.00\n  0.9 1.0\n", "H 0\nS 1 1.00\n  0.5 1.0\n"),
}


def basis(name):
    he, h = BASES[name]
    mol = Molecule.from_angstrom([("He", 0.0, 0.0, 0.0), ("H", 0.3, -0.2, 0.9)])
    return BasisSet.build(mol, parse_gbs("****\n%s****\n%s****\n" % (he, h)))


def split_precision(build):
    """build(cutoff) -> (outputs, stats) at the largest power of ten below which
    some quartets, but not all, run in FP32."""
    for k in range(1, -13, -1):
        out, s = build(10.0 ** k)
        if s["fp64"] > 0:
            break
    assert s["fp32"] > 0 and s["fp64"] > 0
    assert s["fp32"] + s["fp64"] + s["screened"] == s["total"]
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ctype", [LLSS, SSSS])
@pytest.mark.parametrize("name", sorted(BASES))
def test_engine_rel(name, ctype, precision):
    bs = basis(name)
    N = bs.nbasis
    _D, X = rel_inputs(N, 61)
    ref = O.OracleBasis(bs).rel_contract(X, ctype, True)
    c = GTODirectRelERIContraction(DirectTPI(bs))

    def build(cutoff):
        lst = [TwoBodyContraction(X[m], np.zeros((N, N), complex)) for m in range(17)]
        c.twoBodyContract(lst, ctype, precision=precision, fp32_cutoff=cutoff)
        return lst, c.last_stats

    lst = build(0.0)[0] if precision == "fp64" else split_precision(build)
    assert precision == "mixed" or c.last_stats["fp32"] == 0
    for m in OUTS[ctype]:
        assert max_rel(lst[m].AX, ref[m]) < (1e-11 if precision == "fp64" else 1e-6), m


@pytest.mark.parametrize("kind", ["real", "real_nonher", "complex", "complex_nonher", "mixed"])
@pytest.mark.parametrize("name", ["f2", "long", "mix"])
def test_engine_jk(name, kind):
    """J and K of bases with f shells, and of long contractions whose quartets
    several lanes of the class kernels share: every Hermitian / complex flavour and
    mixed precision (three matrices a call)."""
    bs = basis(name)
    N = bs.nbasis
    rng = np.random.default_rng(62)
    cplx, her = kind.startswith("complex"), not kind.endswith("nonher")
    mats = []
    for _ in range(3):
        A = 0.1 * rng.standard_normal((N, N))
        if cplx:
            A = A + 0.1j * rng.standard_normal((N, N))
        mats.append(np.asfortranarray(A + A.conj().T if her else A))
    types = [COULOMB, EXCHANGE, EXCHANGE]
    ref = O.OracleBasis(bs).contract(mats, [int(her)] * 3, types)
    c = GTODirectTPIContraction(DirectTPI(bs))

    def build(cutoff):
        out = [np.zeros((N, N), mats[0].dtype, order="F") for _ in mats]
        c.twoBodyContract([TwoBodyContraction(m, o, her, t) for m, o, t in zip(mats, out, types)],
                          precision="mixed" if kind == "mixed" else "fp64", fp32_cutoff=cutoff)
        return out, c.last_stats

    out = split_precision(build) if kind == "mixed" else build(0.0)[0]
    for o, r in zip(out, ref):
        assert max_rel(o, np.asarray(r)) < (1e-6 if kind == "mixed" else 1e-11)


@pytest.mark.parametrize("name", ["long", "mix"])
def test_jk_without_screen(name):
    """Quartets are shared by lanes without the screen as well."""
    bs = basis(name)
    N = bs.nbasis
    A = 0.1 * np.random.default_rng(66).standard_normal((N, N))
    D = np.asfortranarray(A + A.T)
    ref = O.OracleBasis(bs).contract([D, D], [1, 1], [0, 1], screen=False)
    lst = [TwoBodyContraction(D, np.zeros((N, N), order="F"), True, t)
           for t in (COULOMB, EXCHANGE)]
    c = GTODirectTPIContraction(DirectTPI(bs))
    c.twoBodyContract(lst, screen=False)
    assert c.last_stats["screened"] == 0
    for m, r in zip(lst, ref):
        assert max_rel(m.AX, np.asarray(r)) < 1e-11


@pytest.mark.parametrize("name", sorted(BASES))
def test_engine_gaunt(name):
    bs = basis(name)
    N = bs.nbasis
    _D, X = gaunt_inputs(N, 63)
    ref = O.OracleBasis(bs).rel_contract(X, GAUNT, True)
    lst = [TwoBodyContraction(X[m], np.zeros((N, N), complex)) for m in range(29)]
    GTODirectRelERIContraction(DirectTPI(bs)).twoBodyContract(lst, GAUNT)
    for m in OUTS_X + OUTS_C:
        assert max_rel(lst[m].AX, ref[m]) < 1e-11, m


@pytest.mark.parametrize("name", sorted(BASES))
def test_engine_gradient(name):
    """J and K gradient contractions: two atoms share a quartet in every
    arrangement, the quartets of one atom drop out."""
    bs = basis(name)
    N = bs.nbasis
    rng = np.random.default_rng(64)
    A = rng.standard_normal((N, N))
    D = 0.1 * (A + A.T)
    atoms = np.array([s.atom for s in bs.shells], dtype=np.int32)
    ref = O.OracleBasis(bs).grad_contract([D, D], [O.COULOMB, O.EXCHANGE], atoms, 2)
    cl = [[TwoBodyContraction(D, np.zeros((N, N), order="F"), True, t)
           for t in (COULOMB, EXCHANGE)] for _ in range(6)]
    DirectGradContraction(DirectTPI(bs)).gradTwoBodyContract(cl, atoms)
    for g in range(6):
        for m in range(2):
            assert max_rel(cl[g][m].AX, np.asarray(ref[g][m])) < 1e-11, (g, m)


def test_long_contraction_in_rows():
    """1156 primitive pairs of one shell pair: more than the grids of the set-up
    kernels have rows (PRIM_ROWS)."""
    gbs = "****\nH 0\nS 34 1.00\n" + "".join("  %g %g\n" % (0.1 * 1.3 ** k, 0.1 + 0.01 * k)
                                              for k in range(34)) + "F 1 1.00\n  0.8 1.0\n****\n"
    bs = BasisSet.build(Molecule.from_angstrom([("H", 0.1, 0.2, 0.3)]), parse_gbs(gbs))
    N = bs.nbasis
    A = 0.1 * np.random.default_rng(67).standard_normal((N, N))
    D = np.asfortranarray(A + A.T)
    ref = O.OracleBasis(bs).contract([D, D], [1, 1], [0, 1])
    lst = [TwoBodyContraction(D, np.zeros((N, N), order="F"), True, t)
           for t in (COULOMB, EXCHANGE)]
    GTODirectTPIContraction(DirectTPI(bs)).twoBodyContract(lst)
    for m, r in zip(lst, ref):
        assert max_rel(m.AX, np.asarray(r)) < 1e-11


@pytest.mark.parametrize("count", [32, 33])
def test_many_matrices_share_outputs(count):
    """Device matrices in batches of 32 launches; every contraction adds into
    one J, half of the exchanges into one K, so each is the sum of its parts."""
    torch = pytest.importorskip("torch")
    bs = basis("one")
    N = bs.nbasis
    tpi = DirectTPI(bs)
    rng = np.random.default_rng(71)
    Ds = [d + d.T for d in rng.normal(size=(count, N, N))]
    dev = [torch.tensor(d, device="cuda").T for d in Ds]
    zero = lambda: torch.zeros((N, N), dtype=torch.float64, device="cuda").T
    J, K, L = zero(), zero(), zero()
    lst = []
    for k, d in enumerate(dev):
        lst.append(TwoBodyContraction(d, J, True, COULOMB))
        lst.append(TwoBodyContraction(d, K if k % 2 else L, True, EXCHANGE))
    GTODirectTPIContraction(tpi).twoBodyContract(lst)
    torch.cuda.synchronize()
    refs = [[], []]
    for d in Ds:
        r = [TwoBodyContraction(np.asfortranarray(d), np.zeros((N, N), order="F"), True, t)
             for t in (COULOMB, EXCHANGE)]
        GTODirectTPIContraction(tpi).twoBodyContract(r)
        for t in range(2):
            refs[t].append(r[t].AX)
    # sums of 64 or 66 numbers of one size in another order
    for got, ref in ((J, sum(refs[0])), (K, sum(refs[1][1::2])), (L, sum(refs[1][::2]))):
        scale = max(np.abs(m).max() for t in refs for m in t)
        assert np.abs(got.cpu().numpy() - ref).max() < 1e-13 * count * scale


def ring_basis():
    """24 centres with an s of 7 and an f of 3 primitives: 5400 words in
    (ss|fs), whose items fill the launch stream's region, and (fs|fs) in two
    slabs."""
    t = 2 * np.pi * np.arange(24) / 24
    mol = Molecule.from_angstrom([("H", 2 * np.cos(a), 2 * np.sin(a), 0.3 * (i % 2))
                                  for i, a in enumerate(t)])
    gbs = "****\nH 0\nS 7 1.00\n" + "".join("  %g %g\n" % (0.12 * 2.2 ** k, 0.2 + 0.05 * k)
                                             for k in range(7))
    gbs += "F 3 1.00\n  0.5 0.5\n  1.05 0.5\n  2.205 0.5\n****\n"
    return BasisSet.build(mol, parse_gbs(gbs))


def test_engine_items_fill_region():
    """Words with FP64 and FP32 quartets share the items of their word: a mixed
    build whose items fill the region equals the FP64 build, and both the
    oracle's integrals summed over whole shell blocks without a screen (some 2e3
    quartets a block, each within 1e-12 / 2 of its screened value)."""
    bs = ring_basis()
    N = bs.nbasis
    rng = np.random.default_rng(3)
    A = rng.standard_normal((N, N))
    D = np.asfortranarray(0.1 * (A + A.T))
    res = {}
    for prec in ("fp64", "mixed"):
        c = GTODirectTPIContraction(DirectTPI(bs))
        lst = [TwoBodyContraction(D, np.zeros((N, N), order="F"), True, t)
               for t in (COULOMB, EXCHANGE)]
        c.twoBodyContract(lst, precision=prec, fp32_cutoff=1e-4)
        res[prec] = [m.AX for m in lst]
    assert c.last_stats["fp32"] > 3e5 and c.last_stats["fp64"] > 3e5
    for a, b in zip(res["mixed"], res["fp64"]):
        assert max_rel(a, b) < 1e-6
    ob = O.OracleBasis(bs)
    sl = [slice(o, o + s.size) for o, s in zip(bs.offsets, bs.shells)]
    f = [s for s in range(bs.nshell) if bs.shells[s].l == 3]
    o = [s for s in range(bs.nshell) if bs.shells[s].l == 0]
    for a, b in ((f[0], o[0]), (o[20], o[2])):
        J = K = 0.0
        for c in range(bs.nshell):
            for d in range(bs.nshell):
                if d <= c:
                    g = ob.eri_quartet(a, b, c, d)
                    w = D[sl[c], sl[d]] * (1.0 if c == d else 2.0)
                    J = J + np.einsum("abcd,cd->ab", g, w)
                K = K + np.einsum("acbd,cd->ab", ob.eri_quartet(a, c, b, d), D[sl[c], sl[d]])
        for got, ref in zip(res["fp64"], (J, K)):
            assert np.abs(got[sl[a], sl[b]] - ref).max() < 1e-11 * np.abs(got).max() + 2e-9


@pytest.mark.parametrize("limit", ["0", "0.25"])
def test_windows_of_tables(limit, monkeypatch):
    """Tables beyond the basis' limit: launches build windows of them, of one
    pair at the smallest (every bra pair against every ket pair by itself)."""
    monkeypatch.setenv("CQF_TABLE_LIMIT_MB", limit)
    for name in ("f2", "mix"):
        for kind in ("real", "complex_nonher", "mixed"):
            test_engine_jk(name, kind)
        for ctype in (LLSS, SSSS):
            test_engine_rel(name, ctype, "fp64")
        test_engine_gaunt(name)
        test_engine_gradient(name)


def test_windows_under_capture(monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("CQF_TABLE_LIMIT_MB", "0")
    bs = basis("mix")
    N = bs.nbasis
    rng = np.random.default_rng(81)
    A = 0.1 * rng.standard_normal((N, N))
    X = torch.tensor(A + A.T, device="cuda").T
    out = torch.zeros((2, N, N), dtype=torch.float64, device="cuda")
    graph = ContractionGraph(DirectTPI(bs), [TwoBodyContraction(X, out[k].T, True, t)
                                             for k, t in enumerate((COULOMB, EXCHANGE))])
    for _ in range(2):
        B = 0.1 * rng.standard_normal((N, N))
        X.copy_(torch.tensor(B + B.T))
        out.zero_()
        torch.cuda.synchronize()
        graph.launch()
        torch.cuda.synchronize()
        ref = O.OracleBasis(bs).contract([np.asfortranarray(B + B.T)] * 2, [1, 1], [0, 1])
        for k in range(2):
            assert max_rel(out[k].T.cpu().numpy(), np.asarray(ref[k])) < 1e-11


def test_windows_beyond_fixed_scratch(monkeypatch):
    """The windows of 43 MiB of tables with a limit of 40 (six of 5 MiB) do not
    fit the no-alloc entry point's 32 MiB beside the matrices: it takes the generic
    kernel."""
    monkeypatch.setenv("CQF_TABLE_LIMIT_MB", "40")
    bs = BasisSet.build(workloads.water_cluster(7, seed=3, box=5.0), "cc-pvtz")
    tpi, N = DirectTPI(bs), bs.nbasis
    A = 0.1 * np.random.default_rng(82).standard_normal((N, N))
    D = np.asfortranarray(A + A.T)
    res = []
    for entry in (_cabi.lib().cqf_two_body_contract, _cabi.lib().cqf_two_body_contract_noalloc):
        out = [np.zeros((N, N), order="F") for _ in range(2)]
        assert noalloc_contract(entry, tpi, D, out, [COULOMB, EXCHANGE]) == _cabi.CQF_OK
        res.append(out)
    for a, b in zip(*res):
        assert max_rel(a, b) < 1e-11
