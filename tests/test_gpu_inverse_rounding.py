"""The rounding of the blocked elimination. The levels of a long molecule are so sharp that the last bits of
its Dyson matrices' inverses come back 10^5 times larger in its spectra: an elimination that does other operations,
or the same ones in another order, gives other results to 1e-9, none of them wrong. So the kernels do, on every value,
the operations of the elimination with row exchanges in panels of 16 columns, whatever the order in which they hold and
visit the values. Here that elimination is done in NumPy with exactly rounded multiply-adds: equal bits, without
a tolerance."""
import numpy as np
import pytest

import quichotte_b200 as qb

PB = 16


def two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def split(a):
    c = 134217729.0 * a
    h = c - (c - a)
    return h, a - h


def fma(a, b, c):
    """a b + c rounded once (Boldo and Melquiond, Emulation of FMA and correctly rounded sums, 2008)."""
    uh = a * b
    (ah, al), (bh, bl) = split(a), split(b)
    ul = ((ah * bh - uh) + ah * bl + al * bh) + al * bl
    th, tl = two_sum(c, ul)
    vh, vl = two_sum(uh, th)
    # tl + vl rounded to odd: the neighbour towards the rest where the sum is inexact and even
    z, r = two_sum(tl, vl)
    z = np.array(z, np.float64, ndmin=1)
    bits = z.view(np.int64)
    even = (r != 0.0) & (bits & 1 == 0)
    bits[even] += np.where((r > 0) == (z > 0), 1, -1)[even]
    return np.reshape(vh + z.reshape(np.shape(vh)), np.shape(vh))


def cmul(ax, ay, bx, by):
    return fma(ax, bx, -(ay * by)), fma(ax, by, ay * bx)


def eliminate(A):
    """The inverse of A as the kernels form it."""
    N = len(A)
    X, Y = A.real.copy(), A.imag.copy()
    perm = []
    for k0 in range(0, N, PB):
        K = slice(k0, min(k0 + PB, N))
        for k in range(k0, K.stop):
            p = k + int(np.argmax(np.abs(X[k:, k]) + np.abs(Y[k:, k])))
            perm.append(p)
            for M in (X, Y):
                M[[k, p]] = M[[p, k]]
            # 1 / pivot, its larger part scaled to [1, 2)
            s = 2.0 ** -np.floor(np.log2(max(abs(X[k, k]), abs(Y[k, k]))))
            px, py = X[k, k] * s, Y[k, k] * s
            d = s / fma(px, px, py * py)[()]
            sx, sy = cmul(X[k, K], Y[k, K], px * d, -py * d)
            sx[k - k0], sy[k - k0] = px * d, -py * d
            fx, fy = X[:, k:k + 1].copy(), Y[:, k:k + 1].copy()
            X[:, k] = Y[:, k] = 0.0
            x = fma(fy, sy, fma(-fx, sx, X[:, K]))
            y = fma(-fy, sx, fma(-fx, sy, Y[:, K]))
            x[k], y[k] = sx, sy
            X[:, K], Y[:, K] = x, y
        J = np.r_[0:k0, K.stop:N]
        bx, by = X[K][:, J].copy(), Y[K][:, J].copy()
        cx, cy = X[:, J], Y[:, J]
        cx[K] = cy[K] = 0.0
        ax, ay = X[:, K], Y[:, K]
        for t in range(K.stop - k0):
            cx = fma(ax[:, t:t + 1], bx[t], cx)
            cy = fma(ax[:, t:t + 1], by[t], cy)
        for t in range(K.stop - k0):
            cx = fma(ay[:, t:t + 1], -by[t], cx)
            cy = fma(ay[:, t:t + 1], bx[t], cy)
        X[:, J], Y[:, J] = cx, cy
    for k in range(N - 1, -1, -1):
        for M in (X, Y):
            M[:, [k, perm[k]]] = M[:, [perm[k], k]]
    return X + 1j * Y


def dyson_matrix(N, seed):
    """A matrix close to a level: condition about 1e8."""
    rng = np.random.default_rng(seed)
    H = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    H = (H + H.conj().T) / np.sqrt(2 * N)
    e = np.linalg.eigvalsh(H)[N // 3]
    return (e + 1e-8j) * np.eye(N) - H


def test_reference_elimination_inverts():
    rng = np.random.default_rng(2)
    a, b, c = rng.standard_normal((3, 20000)) * 10.0 ** rng.integers(-3, 4, (3, 20000))
    from fractions import Fraction as F
    for q in range(0, 20000, 40):
        assert fma(a[q:q + 1], b[q:q + 1], c[q:q + 1])[0] == float(F(a[q]) * F(b[q]) + F(c[q]))
    for N in (1, 5, 16, 17, 48):
        A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
        ref = np.linalg.inv(A)
        assert np.max(np.abs(eliminate(A) - ref)) < 1e-11 * np.max(np.abs(ref))


# the matrices above 80 states go to one of two kernels, by their number: 148 and 149 are the two sides
CASES = [(1, 3), (5, 9), (8, 3), (15, 5), (16, 5), (17, 5), (24, 700), (25, 3), (31, 3), (32, 3), (33, 3), (40, 3), (48, 900), (63, 3),
         (64, 3), (65, 3), (80, 3), (81, 148), (81, 149), (88, 149), (95, 149), (96, 148), (96, 149), (97, 148), (97, 149), (113, 149),
         (119, 149), (120, 148), (120, 149), (120, 700), (121, 5), (128, 500), (129, 3), (161, 3), (192, 400), (255, 3), (256, 320)]


@pytest.mark.gpu
@pytest.mark.parametrize("N, batch", CASES)
def test_inverse_has_the_bits_of_the_elimination_with_row_exchanges(N, batch):
    rng = np.random.default_rng(N)
    # sharp levels, dense pivoting, and small whole numbers: columns with many equal candidates
    kinds = [dyson_matrix(N, N), rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)),
             rng.integers(-2, 3, (N, N)) + 1j * rng.integers(-2, 3, (N, N)) + 0.25 * np.eye(N)]
    A = np.array([kinds[b % 3] for b in range(batch)])
    inv, info = qb.invert_batched(A)
    assert not info.any()
    for q, M in enumerate(kinds):
        ref = eliminate(M)
        assert all(np.array_equal(inv[b], ref) for b in range(q, batch, 3)), (q, np.max(np.abs(inv[q] - ref)) / np.max(np.abs(ref)))
