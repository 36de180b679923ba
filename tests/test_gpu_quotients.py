"""The quotients of the FP64 factorisations and solves, which are products by a reciprocal (wb_tri.cuh): where
one division makes a result, it is as close as Smith's."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _random(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * 2.0 ** rng.integers(-200, 200, shape)


def _check(got, num, den):
    num, den = num.astype(np.clongdouble), den.astype(np.clongdouble)
    want = num * den.conj() / (den.real ** 2 + den.imag ** 2)
    err = np.abs((got - want) / want).astype(float) / U
    # a reciprocal off by 1.2 units with its residual's rounding, a complex product of two rounded terms off by 2
    assert err.max() <= 4.0 and np.sqrt((err ** 2).mean()) <= 0.9, (err.max(), np.sqrt((err ** 2).mean()))


# n = 9 and 66: one block and two; 3 and 6 columns: the few-column solve, 8 and 70: the blocked one
@pytest.mark.parametrize('n', [9, 66])
@pytest.mark.parametrize('columns,trans', [(3, 0), (6, 0), (8, 0), (70, 0), (70, 1)])
def test_a_diagonal_system(n, columns, trans):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from device_ops import load
    rng = np.random.default_rng(n + columns)
    batch = 64
    d, b = _random(rng, batch, n), _random(rng, batch, columns, n)
    lu = np.zeros((batch, n, n), complex)
    lu[:, np.arange(n), np.arange(n)] = d
    lu, x = torch.as_tensor(lu).cuda(), torch.as_tensor(b.copy()).cuda()
    piv = torch.arange(n, dtype=torch.int32, device='cuda').expand(batch, n).contiguous()
    assert load().ops_getrs(1, batch, n, lu.data_ptr(), n * n, piv.data_ptr(), x.data_ptr(), columns, trans) == 0
    torch.cuda.synchronize()
    _check(x.cpu().numpy(), b, np.broadcast_to(d[:, None], b.shape))


@pytest.mark.parametrize('n', [20, 65, 130])
def test_the_multipliers_of_a_lower_triangle(n):
    """No element above the diagonal: the factor below it is one division a column"""
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from device_ops import load
    rng = np.random.default_rng(n)
    batch = 20
    s = 2.0 ** rng.integers(-200, 200, (batch, 1, n))
    A = np.tril(rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n)))
    k = np.arange(n)
    A[:, k, k] *= 100.0 / np.abs(A[:, k, k])                          # no interchanges
    A = A * s
    lu = torch.as_tensor(np.ascontiguousarray(A.transpose(0, 2, 1))).cuda()
    piv = torch.zeros((batch, n), dtype=torch.int32, device='cuda')
    st = torch.zeros(batch, dtype=torch.int32, device='cuda')
    assert load().ops_getrf(1, batch, n, lu.data_ptr(), n * n, piv.data_ptr(), st.data_ptr()) == 0
    torch.cuda.synchronize()
    assert int(st.sum()) == 0 and (piv.cpu().numpy() == k).all()
    got = lu.cpu().numpy().transpose(0, 2, 1)
    low = np.tril(np.ones((n, n), bool), -1)
    _check(got[:, low], A[:, low], np.broadcast_to(A[:, None, k, k], A.shape)[:, low])
