"""The few-column solves (getrs_narrow_kernel, wb_tri.cuh) by themselves, at the sizes where the cluster a
matrix gets grows: the same bits for every batch, so for every cluster, and the answer held to its system."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu


def _factor(ops, A, batch):
    n = A.shape[0]
    lu = A.T.contiguous().expand(batch, n, n).contiguous()            # column-major
    piv = torch.zeros((batch, n), dtype=torch.int32, device='cuda')
    st = torch.zeros(batch, dtype=torch.int32, device='cuda')
    assert ops.ops_getrf(int(A.dtype == torch.complex128), batch, n, lu.data_ptr(), n * n, piv.data_ptr(), st.data_ptr()) == 0
    assert int(st.sum()) == 0
    return lu, piv


# n on both sides of 64, 128, 256 (FP64: clusters of 2, 4, 8) and 480, 960 (FP32: 2, 4)
@pytest.mark.parametrize('n', [63, 64, 66, 130, 256, 450, 490, 961])
@pytest.mark.parametrize('dtype', [torch.complex128, torch.complex64])
def test_narrow_solves_keep_their_bits_over_clusters(n, dtype):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from device_ops import load
    ops = load()
    g = torch.Generator(device='cpu').manual_seed(n)
    A = torch.complex(torch.randn((n, n), generator=g, dtype=torch.float64),
                      torch.randn((n, n), generator=g, dtype=torch.float64)).to(dtype).cuda()
    full = torch.complex(torch.randn((n, 6), generator=g, dtype=torch.float64),
                         torch.randn((n, 6), generator=g, dtype=torch.float64)).to(dtype).cuda()
    unit = 2.3e-16 if dtype == torch.complex128 else 1.2e-7
    for k in (1, 3, 6):
        ref = None
        for batch in (1, 30, 80, 200):                                 # clusters of up to 8, 4, 1 and 1 CTAs
            lu, piv = _factor(ops, A, batch)
            x = full[:, :k].T.contiguous().expand(batch, k, n).contiguous()
            assert ops.ops_getrs(int(dtype == torch.complex128), batch, n, lu.data_ptr(), n * n, piv.data_ptr(),
                                 x.data_ptr(), k, 0) == 0
            torch.cuda.synchronize()
            if ref is None:
                ref = x[0].clone()
                wide = lu[0].T.to(torch.complex128)
                mag = (torch.tril(wide.abs(), -1) + torch.eye(n, device='cuda', dtype=torch.float64)) @ torch.triu(wide.abs())
                xw = x[0].T.to(torch.complex128)
                res = (A.to(torch.complex128) @ xw - full[:, :k].to(torch.complex128)).abs()
                # LU with partial pivoting and two substitutions, complex: 3 gamma_n |L| |U| |x|, rows permuted alike
                assert res.max() <= 3 * 4 * n * unit * (mag @ xw.abs()).max()
            assert all(torch.equal(x[p], ref) for p in (0, batch // 2, batch - 1)), (k, batch)


# the largest matrices whose X the kernel holds (200 KB) and one past it: 6 and 3 columns of 16 bytes, 6 of 8
@pytest.mark.parametrize('n,k,dtype', [(2133, 6, torch.complex128), (2134, 6, torch.complex128), (3292, 3, torch.complex128),
                                       (4266, 3, torch.complex128), (4267, 3, torch.complex128), (4266, 6, torch.complex64)])
def test_largest_narrow_solves(n, k, dtype):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from device_ops import load
    ops = load()
    g = torch.Generator(device='cuda').manual_seed(n)
    A = torch.complex(*(torch.randn((n, n), generator=g, dtype=torch.float64, device='cuda') for _ in range(2))).to(dtype)
    b = torch.complex(*(torch.randn((n, k), generator=g, dtype=torch.float64, device='cuda') for _ in range(2))).to(dtype)
    unit = 2.3e-16 if dtype == torch.complex128 else 1.2e-7
    lu, piv = _factor(ops, A, 1)
    x = b.T.contiguous()
    assert ops.ops_getrs(int(dtype == torch.complex128), 1, n, lu.data_ptr(), n * n, piv.data_ptr(), x.data_ptr(), k, 0) == 0
    torch.cuda.synchronize()
    m = lu[0].T.to(torch.complex128).abs()
    mag = (torch.tril(m, -1) + torch.eye(n, device='cuda', dtype=torch.float64)) @ (torch.triu(m) @ x.T.to(torch.complex128).abs())
    res = (A.to(torch.complex128) @ x.T.to(torch.complex128) - b.to(torch.complex128)).abs()
    assert res.max() <= 3 * 4 * n * unit * mag.max()
