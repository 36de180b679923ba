"""The FP64 products by exact slices (wavebit_gb300/csrc/wb_oz.cuh) restated in integers: the scaling of a
panel's lines and of its k, the fixed-point digits, the kept products and their assembly, against exact
rational sums."""
from fractions import Fraction

import numpy as np
import pytest

NONE = None
DROP = 100000


def parts(x):
    """(biased exponent, a subnormal's by its leading bit, None for zero; 53-bit mantissa with sign) of a double"""
    b = int(np.float64(x).view(np.uint64))
    e, m = b >> 52 & 0x7ff, b & (1 << 52) - 1
    if e:
        m |= 1 << 52
    elif m:
        e = m.bit_length() - 52
        m <<= 1 - e
    else:
        e = NONE
    return e, -m if b >> 63 else m


def scales(A, B):
    """Line exponents of A's rows and B's columns and the shift of every k, as zgemm_kernel finds them"""
    K = A.shape[1]
    ea = [[parts(x)[0] for x in row] for row in A]
    eb = [[parts(x)[0] for x in row] for row in B.T]

    def largest(lines, shift):
        return [max((e + s for e, s in zip(l, shift) if e is not NONE and s > -DROP), default=NONE) for l in lines]

    def falls(lines):
        tops = largest(lines, [0] * K)
        return [max((l[k] - t for l, t in zip(lines, tops) if l[k] is not NONE), default=NONE) for k in range(K)]

    fa, fb = falls(ea), falls(eb)
    sa = [-DROP if a is NONE or b is NONE else (b - a) >> 1 for a, b in zip(fa, fb)]
    sb = [-DROP if s == -DROP else -s for s in sa]
    return largest(ea, sa), largest(eb, sb), sa, sb


def fixed(x, top):
    """x in fixed point, 62 bits below 2^(top + 1)"""
    e, m = parts(x)
    if m == 0 or e - top + 9 < -54:
        return 0
    sh = e - top + 9
    if sh >= 0:
        return m << sh
    r = (abs(m) + (1 << -sh - 1)) >> -sh
    return -r if m < 0 else r


def digits(q):
    u = (q + 0x8080808080808080) % 2**64
    return [(u >> 8 * (7 - i) & 0xff) - 128 for i in range(8)]


def assemble(acc, ea, eb):
    """sum acc[w] 256^(7 - w), times 2^(ea + eb) in biased exponents, rounded once (halves away from zero;
    below the normal range too)"""
    h = l = 0
    for w in range(4):
        h, l = h * 256 + acc[w], l * 256 + acc[w + 4]
    total = h * 2**32 + l
    if total == 0:
        return 0.0
    h += l >> 32
    lo = l % 2**32
    neg = h < 0
    if neg:
        h = -h
        if lo:
            h, lo = h - 1, 2**32 - lo
    shift = 0
    if h == 0:
        h, lo, shift = lo, 0, 32
    n = 64 - h.bit_length()
    m = h << n | (lo << n - 32 if n >= 32 else lo >> 32 - n)
    e = ea + eb - n - 994 - shift
    drop = 11 + (1 - e if e < 1 else 0)
    if drop > 64:
        return 0.0
    r = (m >> drop) + (m >> drop - 1 & 1)
    if r == 0:
        return 0.0
    if e < 1:
        bits = r
    else:
        if r >> 53:
            r, e = r >> 1, e + 1
        if e >= 2047:
            return -np.inf if neg else np.inf
        bits = e << 52 | r & 2**52 - 1
    return float(np.uint64(bits | int(neg) << 63).view(np.float64))


def product(A, B):
    ta, tb, sa, sb = scales(A, B)
    M, K = A.shape
    N = B.shape[1]
    C = np.zeros((M, N))
    da = [[digits(fixed(A[i, k], ta[i] - sa[k])) if ta[i] is not NONE else [0] * 8 for k in range(K)] for i in range(M)]
    db = [[digits(fixed(B[k, j], tb[j] - sb[k])) if tb[j] is not NONE else [0] * 8 for k in range(K)] for j in range(N)]
    for i in range(M):
        for j in range(N):
            acc = [0] * 8
            for k in range(K):
                for w in range(8):
                    acc[w] += sum(da[i][k][t] * db[j][k][w - t] for t in range(w + 1))
            assert max(map(abs, acc)) <= 2**24
            if ta[i] is not NONE and tb[j] is not NONE:
                C[i, j] = assemble(acc, ta[i], tb[j])
    return C


def exact(A, B):
    S = [[sum(Fraction(A[i, k]) * Fraction(B[k, j]) for k in range(A.shape[1])) for j in range(B.shape[1])]
         for i in range(A.shape[0])]
    G = [[sum(abs(Fraction(A[i, k]) * Fraction(B[k, j])) for k in range(A.shape[1])) for j in range(B.shape[1])]
         for i in range(A.shape[0])]
    return S, G


def worst(A, B):
    """largest |C - exact| over sum |a||b|, in units of 2^-53"""
    C = product(A, B)
    S, G = exact(A, B)
    return max(float(abs(Fraction(C[i, j]) - S[i][j]) / G[i][j]) * 2**53 for i in range(len(S)) for j in range(len(S[0])))


def entries(rng, *shape):
    """+-[1/2, 2)"""
    return rng.uniform(0.5, 2.0, shape) * rng.choice([-1.0, 1.0], shape)


# An entry keeps 2^-62 of its line's largest and the dropped pairs are below 2^-57 of the two lines' largest,
# K terms of them; with entries of [1/2, 2) and the k's shift one binary order off at most, that is below one
# unit of 2^-53 of sum |a||b|; the one rounding is another.
@pytest.mark.parametrize('K', [1, 8, 64])
def test_dense_products_to_a_rounding(K):
    rng = np.random.default_rng(K)
    assert worst(entries(rng, 3, K), entries(rng, K, 3)) <= 2.0


@pytest.mark.parametrize('K', [2, 16, 64])
@pytest.mark.parametrize('s', [1, 9, 20, 40, 60])
def test_operands_graded_along_k(K, s):
    """One operand falls by 2^s a term (at most 2^900 in all), the other rises by it: every term counts, as in
    modes scaled by any factors and their inverse."""
    rng = np.random.default_rng(100 * K + s)
    s = min(s, 900 // K)
    g = 2.0 ** (-s * np.arange(K))
    assert worst(entries(rng, 3, K) * g, entries(rng, K, 3) / g[:, None]) <= 2.0
    perm = rng.permutation(K)
    assert worst(entries(rng, 3, K) / g[perm], entries(rng, K, 3) * g[perm, None]) <= 2.0


def test_rows_and_columns_of_any_scale():
    rng = np.random.default_rng(7)
    K = 16
    d = [2.0 ** rng.integers(-300, 300, m) for m in (4, K, 4)]
    assert worst(entries(rng, 4, K) * d[0][:, None] * d[1], entries(rng, K, 4) / d[1][:, None] * d[2]) <= 2.0


def test_one_wild_row_leaves_the_others_alone():
    rng = np.random.default_rng(8)
    A, B = entries(rng, 4, 16), entries(rng, 16, 4)
    A[0] *= 2.0 ** np.concatenate([[300], np.full(15, 200)])
    C, (S, G) = product(A, B), exact(A, B)
    for i in range(1, 4):
        for j in range(4):
            assert abs(Fraction(C[i, j]) - S[i][j]) <= 2 * G[i][j] / 2**53
    # row 0: 2^-57 of the lines' largest a term, never worse than without the shifts
    for j in range(4):
        assert abs(Fraction(C[0, j]) - S[0][j]) <= 2 * G[0][j] / 2**53


def test_zeros_and_the_ends_of_the_range():
    rng = np.random.default_rng(9)
    A, B = entries(rng, 4, 8), entries(rng, 8, 4)
    A[0] = 0.0
    A[:, 3] = 0.0
    B[3] *= 2.0 ** 900                                    # meets zeros only
    B[:, 1] = 0.0
    assert not product(A, B)[0].any() and not product(A, B)[:, 1].any()
    S, G = exact(A, B)
    C = product(A, B)
    for i in range(1, 4):
        for j in (0, 2, 3):
            assert abs(Fraction(C[i, j]) - S[i][j]) <= 2 * G[i][j] / 2**53
    tiny = 5e-324
    # subnormal operands and results: to half of the smallest number and a rounding
    for X, Y in ((A * 2.0 ** -1060, B[:, [0, 2, 3]] * 2.0 ** -910), (A * 2.0 ** -540, B[:, [0, 2, 3]] * 2.0 ** -530),
                 (A * 2.0 ** 511, B[:, [0, 2, 3]]), (A * 2.0 ** 1000, B[:, [0, 2, 3]] * 2.0 ** -1050)):
        Y[3] = 0.0
        S, G = exact(X, Y)
        C = product(X, Y)
        for i in range(4):
            for j in range(3):
                assert abs(Fraction(C[i, j]) - S[i][j]) <= 2 * G[i][j] / 2**53 + Fraction(tiny)


def test_assembly_rounds_once():
    rng = np.random.default_rng(10)
    for t in range(20000):
        acc = [int(v) for v in rng.integers(-2**24, 2**24 + 1, 8)]
        if t % 4 == 0:
            acc[:int(rng.integers(1, 8))] = [0] * 8
            acc = acc[:8]
        total = sum(a * 256 ** (7 - w) for w, a in enumerate(acc))
        got = assemble(acc, 1023, 1023)
        # value: total 256^(7) in digits of 2^-61 each side, 2^(-122) in all: 56 bits are the seven lower weights
        want = Fraction(total) * Fraction(2) ** (56 - 122)
        assert abs(Fraction(got) - want) <= abs(want) / 2**53, (acc, got)
        if total == 0:
            assert got == 0.0
