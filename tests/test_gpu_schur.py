"""The FP64 Schur form by itself: matrices whose eigenvalues coincide (where the sweep stalls and only the rule for
pairs that cannot be told apart deflates), cyclic ones (where the shift stalls) and graded pairs: T upper triangular,
A = Z T Z^H, Z unitary."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu

EPS = 2.3e-16


def _schur(A):
    from device_ops import load
    batch, n, _ = A.shape
    t = torch.as_tensor(np.ascontiguousarray(A.transpose(0, 2, 1))).cuda()
    z, w, tau = torch.zeros_like(t), torch.zeros((batch, n), dtype=t.dtype, device='cuda'), torch.zeros((batch, n), dtype=t.dtype, device='cuda')
    st = torch.zeros(batch, dtype=torch.int32, device='cuda')
    assert load().ops_schur(batch, n, t.data_ptr(), z.data_ptr(), w.data_ptr(), tau.data_ptr(), st.data_ptr()) == 0
    torch.cuda.synchronize()
    return t.cpu().numpy().transpose(0, 2, 1), z.cpu().numpy().transpose(0, 2, 1), w.cpu().numpy(), st.cpu().numpy()


def _unitary(rng, n):
    return np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]


def _matrices(kind, n):
    rng = np.random.default_rng(n)
    out = []
    for t in range(4):
        Q = _unitary(rng, n)
        if kind == 'one value':                          # a multiple of the identity
            A = (1.3 + 0.2j * t) * np.eye(n) + 0j
        elif kind == 'pairs':                            # every eigenvalue twice
            d = np.repeat(rng.standard_normal((n + 1) // 2) + 1j * rng.standard_normal((n + 1) // 2), 2)[:n]
            A = Q @ np.diag(d) @ Q.conj().T
        elif kind == 'two values':
            A = Q @ np.diag(np.where(rng.random(n) < 0.5, 2.0, -1.0 + t)) @ Q.conj().T
        elif kind == 'pairs apart by rounding':
            d = np.repeat(rng.uniform(1, 2, (n + 1) // 2), 2)[:n] * (1 + 2.2e-16 * rng.integers(-2, 3, n))
            A = Q @ np.diag(d) @ Q.conj().T
        elif kind == 'jordan':                           # a large chain of one eigenvalue
            A = Q @ (np.diag(np.full(n, 1.0 + 0j)) + np.diag(np.full(n - 1, 0.5 ** t), 1)) @ Q.conj().T
        elif kind == 'cyclic':
            A = np.roll(np.eye(n), 1, axis=0).astype(complex) * (1 + t)
        else:                                            # 'graded': entries over many orders, no two rows alike
            A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * 10.0 ** (-0.3 * np.arange(n))[:, None]
        out.append(A)
    return np.stack(out).astype(complex)


# n = 20: the element-by-element sweep; 33 and past: the windows of 16 reflectors, one and several
@pytest.mark.parametrize('n', [20, 33, 50, 98, 130])
@pytest.mark.parametrize('kind', ['one value', 'pairs', 'two values', 'pairs apart by rounding', 'jordan', 'cyclic', 'graded'])
def test_schur_form_of_matrices_that_stall(kind, n):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    A = _matrices(kind, n)
    T, Z, w, st = _schur(A)
    # A null space of half the order is a block of rounding noise to the sweep, which may run out of steps on it: such
    # a matrix (the second of 'two values') is then flagged and its unfound eigenvalues are NaN. No other may be.
    out = (st == 2) & (kind == 'two values') & (np.arange(4) == 1)
    assert not st[~out].any(), st
    assert np.isnan(w[out]).any(axis=1).all()
    A, T, Z, w = A[~out], T[~out], Z[~out], w[~out]
    low = np.tril(np.ones((n, n), bool), -1)
    for a, t, z, x in zip(A, T, Z, w):
        t = np.where(low, 0, t)
        assert np.array_equal(np.diag(t), x)
        # reduction and sweeps, each unitary to a few n units; a deflation drops a unit of its diagonal's size
        assert np.abs(z.conj().T @ z - np.eye(n)).max() <= 40 * n * EPS
        assert np.abs(z @ t @ z.conj().T - a).max() <= 40 * n * EPS * np.abs(a).sum(axis=1).max()
