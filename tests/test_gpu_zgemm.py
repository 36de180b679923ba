"""The FP64 products (oz::zgemm_kernel, wb_oz.cuh) by themselves: tiles, panels and chunks at their edges, every
form of call, graded operands, the ends of the range, infinities and NaN, against sums in extended precision."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _entries(rng, *shape, kind=complex):
    """components of +-[1/2, 2)"""
    def real():
        return rng.uniform(0.5, 2.0, shape) * rng.choice([-1.0, 1.0], shape)
    return real() + 1j * real()


def _ll(*v):
    return (ctypes.c_longlong * 3)(*v)


def _store(M, order):
    """(device tensor, strides) of a batch of matrices, by columns ('F'), by rows ('C') or by columns with a gap"""
    b, r, c = M.shape
    if order == 'C':
        t = torch.as_tensor(np.ascontiguousarray(M))
        s = _ll(c, 1, r * c)
    else:
        ld = r + (3 if order == 'gap' else 0)
        buf = np.full((b, c, ld), np.nan + 0j)
        buf[:, :, :r] = M.transpose(0, 2, 1)
        t = torch.as_tensor(buf)
        s = _ll(1, ld, c * ld)
    return t.cuda(), s


def _load(t, s, r, c):
    v = t.cpu().numpy().reshape(t.shape[0], -1)
    i = np.arange(r)[:, None] * s[0] + np.arange(c)[None, :] * s[1]
    return v[:, i]


def _product(A, B, C=None, alpha=1.0, beta=0.0, orders='FFF', idx=None, conj=(False, False)):
    """alpha op(A) op(B) + beta C on the device"""
    from device_ops import load
    batch = len(idx) if idx is not None else A.shape[0]
    m, k, n = A.shape[1], A.shape[2], B.shape[2]
    a, sa = _store(A, orders[0])
    b, sb = _store(B, orders[1])
    c, sc = _store(np.full((batch, m, n), np.nan + 0j) if C is None else C, orders[2])
    di = torch.as_tensor(np.asarray(idx, np.int32)).cuda() if idx is not None else None
    alpha, beta = complex(alpha), complex(beta)
    rc = load().ops_zgemm(batch, m, n, k, alpha.real, alpha.imag, a.data_ptr(), sa, di.data_ptr() if di is not None else None,
                          conj[0], b.data_ptr(), sb, conj[1], beta.real, beta.imag, c.data_ptr(), sc)
    assert rc == 0
    torch.cuda.synchronize()
    return _load(c, sc, m, n)


def _exact(A, B):
    """The product in extended precision and its magnitudes: sum |a||b| over the four real products"""
    L = np.clongdouble
    want = np.einsum('bik,bkj->bij', A.astype(L), B.astype(L))
    mag = np.einsum('bik,bkj->bij', np.abs(A.real) + np.abs(A.imag), np.abs(B.real) + np.abs(B.imag))
    return want, mag


def _cuda():
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')


def _within(got, want, mag, units):
    d = got.astype(np.clongdouble) - want
    assert np.isfinite(got).all()
    worst = max((np.abs(d.real) / mag).max(), (np.abs(d.imag) / mag).max()) / U
    assert worst <= units, float(worst)


# Entries keep 2^-62 of their lines' largest and the dropped pairs are below 2^-57 of the two lines' largest; with
# components in [1/2, 2) that is a unit of sum |a||b| at most. Each panel of 64 rounds its sum, and each addition.
def _units(k):
    return 1 + 2 * -(-k // 64)


@pytest.mark.parametrize('mnk', [(8, 8, 8), (7, 9, 9), (9, 65, 63), (63, 64, 65), (65, 9, 129), (64, 130, 200), (128, 64, 16)])
def test_edges_of_tiles_panels_and_chunks(mnk):
    _cuda()
    m, n, k = mnk
    rng = np.random.default_rng(m * n + k)
    A, B = _entries(rng, 2, m, k), _entries(rng, 2, k, n)
    want, mag = _exact(A, B)
    _within(_product(A, B), want, mag, _units(k) if min(mnk) >= 8 else 2 * k + 2)   # thin: a chain of FMAs
    from wavebit_gb300 import _lib
    assert int(_lib.load().wb_tensor_core_errors()) == 0


@pytest.mark.parametrize('orders', ['FFF', 'CFF', 'FCF', 'CCC', 'gap'])
@pytest.mark.parametrize('conj', [(False, False), (True, False), (False, True), (True, True)])
def test_strides_and_conjugates(orders, conj):
    _cuda()
    rng = np.random.default_rng(len(orders) + 10 * conj[0] + 20 * conj[1])
    A, B = _entries(rng, 2, 66, 70), _entries(rng, 2, 70, 33)
    want, mag = _exact(A.conj() if conj[0] else A, B.conj() if conj[1] else B)
    orders = ('gap',) * 3 if orders == 'gap' else orders
    _within(_product(A, B, orders=orders, conj=conj), want, mag, _units(70))


@pytest.mark.parametrize('alpha,beta', [(1.0, 0.0), (-1.0, 1.0), (0.75, -0.5), (2 - 1j, 1.0), (1.0, 0.5j)])
@pytest.mark.parametrize('indexed', [False, True])
def test_factors_and_indexed_operands(alpha, beta, indexed):
    _cuda()
    rng = np.random.default_rng(int(8 * abs(alpha) + abs(beta)))
    idx = [2, 0, 2, 1] if indexed else None
    A, B = _entries(rng, 3 if indexed else 4, 40, 24), _entries(rng, 4, 24, 65)
    C = _entries(rng, 4, 40, 65)
    want, mag = _exact(A[idx] if indexed else A, B)
    L = np.clongdouble
    want = L(alpha) * want + L(beta) * C.astype(L)
    mag = 2 * abs(alpha) * mag + 2 * abs(beta) * (np.abs(C.real) + np.abs(C.imag))
    # the product's units, the two products by alpha and beta and their sum; complex factors: a chain of FMAs
    _within(_product(A, B, C, alpha, beta, idx=idx), want, mag, 4 + _units(24) + (2 * 24 if complex(alpha).imag or complex(beta).imag else 0))


@pytest.mark.parametrize('s', [1, 9, 20, 40, 60])
@pytest.mark.parametrize('k', [8, 16, 130])
def test_operands_graded_along_k(s, k):
    """One operand falls by 2^s a term, the other rises by it (modes of any normalisation against their inverse)"""
    _cuda()
    rng = np.random.default_rng(100 * k + s)
    g = 2.0 ** -(min(s, 900 // k) * rng.permutation(k))
    A, B = _entries(rng, 1, 70, k), _entries(rng, 1, k, 66)
    want, mag = _exact(A, B)
    _within(_product(A * g, B / g[:, None]), want, mag, _units(k))
    d, f = 2.0 ** rng.integers(-100, 100, 70), 2.0 ** rng.integers(-100, 100, 66)      # all within the normal range
    got = _product(A * g * d[:, None], B / g[:, None] * f)
    _within(got / d[:, None] / f, want, mag, _units(k))


def test_scaled_rows_and_columns_keep_their_bits():
    _cuda()
    rng = np.random.default_rng(3)
    A, B = _entries(rng, 1, 70, 100), _entries(rng, 1, 100, 64)
    d, f = 2.0 ** rng.integers(-300, 300, 70), 2.0 ** rng.integers(-300, 300, 64)
    assert np.array_equal(_product(A * d[:, None], B * f), _product(A, B) * d[:, None] * f)


def test_ends_of_the_range():
    _cuda()
    rng = np.random.default_rng(4)
    A, B = _entries(rng, 1, 20, 24), _entries(rng, 1, 24, 20)
    A[:, 5] = 0.0
    A[:, :, 3] = 0.0
    B[:, :, 7] = 0.0
    want, mag = _exact(A, B)
    B[:, 3] *= 2.0 ** 900                                             # meets zeros only
    got = _product(A, B)
    assert not got[:, 5].any() and not got[:, :, 7].any()
    some = mag > 0
    _within(np.where(some, got, 0), want, np.where(some, mag, 1), _units(24))
    B[:, 3] *= 2.0 ** -900
    for ea, eb in ((-1060, -10), (-530, -530), (511, 500), (1000, -1050)):   # subnormal operands, subnormal and huge results
        X, Y = A * 2.0 ** ea, B * 2.0 ** eb
        want, mag = _exact(X, Y)
        d = _product(X, Y).astype(np.clongdouble) - want
        assert (np.maximum(np.abs(d.real), np.abs(d.imag)) <= _units(24) * U * mag + 5e-324).all(), (ea, eb)
    big = _product(A * 2.0 ** 600, B * 2.0 ** 600)
    assert np.isinf(big.real[some]).all() and np.isinf(big.imag[some]).all() and not big[~some].any()


@pytest.mark.parametrize('value', [np.inf, -np.inf, np.nan])
def test_nonfinite_entries_reach_their_lines_alone(value):
    _cuda()
    rng = np.random.default_rng(5)
    A, B = _entries(rng, 2, 70, 80), _entries(rng, 2, 80, 66)
    clean = _product(A, B)
    A[0, 67, 70] = complex(value, 1.0)
    B[1, 2, 65] = complex(1.0, value)
    got = _product(A, B)
    bad = np.zeros(got.shape, bool)
    bad[0, 67] = bad[1, :, 65] = True
    assert not np.isfinite(got[bad]).any()
    want, mag = _exact(np.where(np.isfinite(A), A, 0), np.where(np.isfinite(B), B, 0))
    _within(np.where(bad, 0, got), np.where(bad, 0, want), mag, _units(80))
    assert np.array_equal(got[0, :64], clean[0, :64])                 # tiles without it keep their bits
