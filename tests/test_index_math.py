"""The index and Pauli-algebra identities the four-component kernels rely on
(csrc/cqf_common.cuh, csrc/cqf_deriv.cuh, csrc/cqf_hgemm.cuh, csrc/cqf_rel.cu),
checked on the host against their definitions: closed-form Cartesian exponents
against the enumeration of the component order, the engine's recursion parents
and cube places against the compact Hermite index, the incremental Hermite index
step, and the Pauli products as permutations against 2 x 2 matrix products."""
import numpy as np


def nherm(L):
    return (L + 1) * (L + 2) * (L + 3) // 6 if L >= 0 else 0


def hidx(t, u, v):
    return nherm(t + u + v - 1) + (u + v) * (u + v + 1) // 2 + v


def cart_row(i):  # cqf_common.cuh
    return sum(i >= tri for tri in (1, 3, 6, 10, 15, 21, 28, 36))


def test_cartesian_exponents_closed_form():
    for l in range(9):
        i = 0
        for a in range(l + 1):
            for b in range(a + 1):  # the libint / CCA component order
                r = cart_row(i)
                lz = i - r * (r + 1) // 2
                assert (l - r, r - lz, lz) == (l - a, a - b, b)
                i += 1


def hg_index(e, S):
    """hg_index (cqf_hgemm.cuh): parents p1, p2, axis and factor of the
    recursion R_h = X_axis R_p1 + cf R_p2, and the cube place."""
    n = 0
    while nherm(n) <= e:
        n += 1
    r = e - nherm(n - 1)
    k = 0
    while (k + 1) * (k + 2) // 2 <= r:
        k += 1
    v = r - k * (k + 1) // 2
    u = k - v
    t = n - k
    p1 = p2 = ax = cf = 0
    if t > 0:
        p1, cf = hidx(t - 1, u, v), t - 1
        p2 = hidx(t - 2, u, v) if t > 1 else 0
    elif u > 0:
        ax, p1, cf = 1, hidx(0, u - 1, v), u - 1
        p2 = hidx(0, u - 2, v) if u > 1 else 0
    elif v > 0:
        ax, p1, cf = 2, hidx(0, 0, v - 1), v - 1
        p2 = hidx(0, 0, v - 2) if v > 1 else 0
    return (t, u, v), p1, p2, ax, cf, (t * S + u) * S + v


def test_engine_hermite_index():
    for L in (0, 1, 3, 16):
        S = L + 1
        at = {}
        for e in range(nherm(L)):
            tuv, p1, p2, ax, cf, off = hg_index(e, S)
            assert hidx(*tuv) == e and off <= L * S * S
            # packed as p1 | p2 << 10 | axis << 20 | factor << 22
            assert p1 < 1024 and p2 < 1024 and cf < 1024
            at[tuv] = off
            if sum(tuv):
                down = list(tuv)
                down[ax] -= 1
                assert p1 == hidx(*down) and cf == down[ax]
                if cf:
                    down[ax] -= 1
                    assert p2 == hidx(*down)
        # the place of h + h' is the sum of theirs
        for a in list(at)[:40]:
            for b in list(at)[::7]:
                c = tuple(x + y for x, y in zip(a, b))
                if sum(c) <= L:
                    assert at[c] == at[a] + at[b]


def test_incremental_hermite_index():
    # hdot_v (cqf_deriv.cuh): hidx(t, u, v + k) by steps
    for t in range(9):
        for u in range(9):
            for v in range(9):
                s = t + u + v
                idx, inc = hidx(t, u, v), (s + 1) * (s + 2) // 2 + (u + v) + 2
                for k in range(9):
                    assert idx == hidx(t, u, v + k)
                    idx += inc
                    inc += s + k + 3


_SIG = [np.eye(2), np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]),
        np.diag([1.0, -1.0])]


def _mat(q):
    return sum(c * s for c, s in zip(q, _SIG))


def _dec(M):
    return np.array([np.trace(M @ s) / 2 for s in _SIG])


def test_pauli_left_and_right_sigma():
    rng = np.random.default_rng(3)
    for _ in range(20):
        t = rng.standard_normal(4) + 1j * rng.standard_normal(4)
        s, x, y, z = t
        # qsig: t sigma_k
        want = [_dec(_mat(t) @ _SIG[k]) for k in (1, 2, 3)]
        got = [np.array([x, s, 1j * z, -1j * y]), np.array([y, -1j * z, s, 1j * x]),
               np.array([z, 1j * y, -1j * x, s])]
        for w, g in zip(want, got):
            assert np.allclose(w, g)
        # left_sigma: i sigma_k t
        want = [_dec(1j * _SIG[k] @ _mat(t)) for k in (1, 2, 3)]
        got = [np.array([1j * x, 1j * s, z, -y]), np.array([1j * y, -z, 1j * s, x]),
               np.array([1j * z, y, -x, 1j * s])]
        for w, g in zip(want, got):
            assert np.allclose(w, g)
        # right_sigmas: sum_b (i f)^[b > 0] t_b sigma_b, f = +-1 (its components
        # are added as (-f im, f re))
        tb = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
        for f in (1.0, -1.0):
            want = _dec(sum((1j * f if b else 1.0) * _mat(tb[b]) @ _SIG[b] for b in range(4)))
            sig = lambda q, k: _dec(_mat(q) @ _SIG[k])
            got = tb[0] + sum(1j * f * sig(tb[b], b) for b in (1, 2, 3))
            assert np.allclose(want, got)
