"""The FP64 kernels at the sizes where their tiles, panels and register blocks begin, end and run over:
the Hessenberg reduction and Q over a cluster, the LU panels and the blocked solves, the few-column
transposed solves, and the products on the tensor cores against the FP64 pipes."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu

EPS = 2.3e-16


def _cuda():
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')


# n = 2 (2 hu + 1): one and two rows a lane (34, 62, 66), four (126, 130), eight (254), the one-column form
# of Q (258), and past what the cluster's shared memory is used for (514)
@pytest.mark.parametrize('hu', [8, 15, 16, 31, 32, 63, 64, 128])
def test_hessenberg_eigenpairs_and_bits_over_clusters(hu):
    _cuda()
    from oracle import rcwa_oracle as O
    from wavebit_gb300 import engine as E
    rng = np.random.default_rng(hu)
    eps = np.where(rng.random((1, 1, 300)) < 0.5, 1.0, 6.0).astype(complex)
    conv = E.assemble(torch.as_tensor(eps, device='cuda'), hu, 0)
    u = np.arange(-hu, hu + 1) * 0.71
    ref = None
    for P in (1, 25, 80) if hu < 63 else (1, 25) if hu < 128 else (1,):       # 8, 4 and 1 CTAs a matrix
        kx, ky = np.tile(u + 0.13, (P, 1)), np.full((P, 2 * hu + 1), 0.21)
        w, q, W, V, st = E.layer_modes(conv, np.zeros(P, int), kx, ky, precision='double')
        assert not (st.cpu().numpy() & ~8).any()
        w, W = w.cpu().numpy(), W.cpu().numpy()
        if ref is None:
            ref = w[0], W[0]
            om2 = O.layer_operator(kx[0], ky[0], *(conv.slot(k)[0].cpu().numpy() for k in range(3)))[0]
            # a Schur form and one triangular solve: a few n units of roundoff of the operator's norm
            res = np.abs(om2 @ W[0] - W[0] * w[0]).max()
            assert res <= 40 * om2.shape[0] * EPS * np.abs(om2).sum(axis=1).max(), res
        for p in (0, P // 2, P - 1):
            assert np.array_equal(w[p], ref[0]) and np.array_equal(W[p], ref[1]), (P, p)


# N = (2 hu + 1)(2 hv + 1) = 9, 33, 35, 63, 65, 99, 129, 225: below a panel, one row past it, one and two
# blocks of 64 and their edges
@pytest.mark.parametrize('orders', [(1, 1), (16, 0), (3, 2), (4, 3), (6, 2), (5, 4), (64, 0), (7, 7)])
@pytest.mark.parametrize('tensor_cores', [True, False])
def test_inverse_of_the_direct_matrix(orders, tensor_cores):
    _cuda()
    from oracle import rcwa_oracle as O
    from wavebit_gb300 import _lib, engine as E
    hu, hv = orders
    rng = np.random.default_rng(3 * hu + hv)
    eps = np.where(rng.random((2, 1 if hv == 0 else 40, 160)) < 0.5, 1.0, 9.0 + 0.3j)
    lib = _lib.load()
    try:
        _lib.check(lib.wb_set_tuning(_lib.WB_TUNE_TENSOR_CORES, 0 if tensor_cores else 1))
        conv = E.assemble(torch.as_tensor(eps, device='cuda'), hu, hv)
        X = conv.slot(2).cpu().numpy()
    finally:
        _lib.check(lib.wb_set_tuning(_lib.WB_TUNE_TENSOR_CORES, 0))
    for l in range(2):
        D = O.conv_matrix(eps[l], hu, hv)
        n = D.shape[0]
        # LU with partial pivoting and two triangular solves: a few n units of roundoff of |X| |D| (and the
        # series of both sides, to a few units themselves)
        bound = 40 * n * EPS * np.abs(X[l]).sum(axis=1).max() * np.abs(D).sum(axis=1).max()
        assert np.abs(X[l] @ D - np.eye(n)).max() <= bound
    assert int(lib.wb_tensor_core_errors()) == 0


# n = 18 (the smallest blocked transposed solve), 30, 50, 70, 98, 162: one to three blocks, equal and ragged
@pytest.mark.parametrize('orders', [(1, 1), (2, 1), (2, 2), (3, 2), (3, 3), (4, 4)])
def test_transposed_solves_of_few_columns(orders):
    _cuda()
    from test_gpu_vjp import _case, _inputs, _modes
    from vjp_case import eff_cotangents, rel, weights
    from wavebit_gb300 import engine
    case = _case(seed=5, L=2, ny=20, nx=22, hu=orders[0], hv=orders[1])
    wR, wT = weights(case, 4)
    _, gW_t, gV_t, gq_t, gth_t = case.stage_c_torch(wR, wT)
    gR, gT = eff_cotangents(case, wR, wT)
    W, V, q = _modes(case)
    gW, gV, gq, gth, st = engine.smm_solve_vjp(W, V, q, _inputs(case), case.hu, case.hv, gR, gT)
    torch.cuda.synchronize()
    assert int(st.abs().sum()) == 0
    # n units of roundoff times the condition of the mode matrices and cascade (up to some 1e4) twice over
    for got, want in ((gW, gW_t), (gV, gV_t), (gq, gq_t), (gth, gth_t)):
        assert rel(got, want) < 1e-9


# n = 50, 98, 242: products of K = 32 .. 242 with ragged tiles of 64
@pytest.mark.parametrize('orders', [(2, 2), (3, 3), (5, 5)])
def test_cascade_with_and_without_tensor_cores(orders):
    _cuda()
    from wavebit_gb300 import _lib, engine as E
    hu, hv = orders
    rng = np.random.default_rng(hu)
    eps = np.where(rng.random((2, 48, 60)) < 0.5, 1.0, 6.0).astype(complex)
    conv = E.assemble(torch.as_tensor(eps, device='cuda'), hu, hv)
    B = 3
    inp = E.BatchInputs([[0, 1]] * B, [[120.0, 90.0]] * B, [700.0, 810.0, 1230.0], [[1000.0, 1000.0]] * B, [0.2] * B,
                        [0.4] * B, [1.0] * B, [2.25] * B, [[0.6 + 0j, 0.8 + 0j]] * B)
    lib = _lib.load()
    out = []
    try:
        for off in (0, 1):
            _lib.check(lib.wb_set_tuning(_lib.WB_TUNE_TENSOR_CORES, off))
            R, T, st = E.solve_batch(conv, inp, precision='double')
            assert not (st.cpu().numpy() & ~8).any()
            out.append((R.cpu().numpy(), T.cpu().numpy()))
    finally:
        _lib.check(lib.wb_set_tuning(_lib.WB_TUNE_TENSOR_CORES, 0))
    assert int(lib.wb_tensor_core_errors()) == 0
    # two FP64 evaluations of the same solve: n units of roundoff times a condition of up to 1e4
    tol = 1e4 * conv.slot(0).shape[-1] * 2 * EPS
    for a, b in zip(out[0], out[1]):
        assert np.abs(a - b).max() <= tol
    for R, T in out:                                     # lossless: every polarization's powers sum to one
        assert np.abs((R + T).sum(axis=(-2, -1)) - 1.0).max() <= 1e3 * tol
