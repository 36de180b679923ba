"""The windowed QR sweep (wb_qr.cuh) at the sizes where its windows (32 reflectors in FP32, 16 in the
16-byte forms) begin, end and run over: eigenpairs by their residual, and the same bits for every
batch size (the CTAs a matrix gets) and thread count."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu

# n = 2 (2 hu + 1)(2 hv + 1): 2, 14, 18, 30 (below a window), 34, 50, 66, 70, 98, 130 (around 1..8 windows)
ORDERS = [(0, 0), (3, 0), (4, 0), (7, 0), (8, 0), (2, 2), (16, 0), (3, 2), (3, 3), (32, 0)]


def _pairs(hu, hv, P):
    from wavebit_gb300 import engine as E
    rng = np.random.default_rng(10 * hu + hv)
    eps = np.where(rng.random((1, 1 if hv == 0 else 24, 60)) < 0.5, 1.0, 6.0).astype(complex)
    conv = E.assemble(torch.as_tensor(eps, device='cuda'), hu, hv)
    u, v = np.arange(-hu, hu + 1) * 0.71, np.arange(-hv, hv + 1) * 0.83
    kx = np.tile(np.tile(u + 0.13, 2 * hv + 1), (P, 1))
    ky = np.tile(np.repeat(v + 0.21, 2 * hu + 1), (P, 1))
    return conv, kx, ky


@pytest.mark.parametrize('orders', ORDERS)
@pytest.mark.parametrize('form', ['double', 'mixed_df64', 'mixed'])
def test_eigenpairs_and_bits_over_batches(orders, form):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from oracle import rcwa_oracle as O
    from wavebit_gb300 import _lib, engine as E
    hu, hv = orders
    lib = _lib.load()
    ref = None
    for P, threads in ((1, 0), (3, 0), (1, 128), (200, 0)):
        conv, kx, ky = _pairs(hu, hv, P)
        try:
            _lib.check(lib.wb_set_tuning(_lib.WB_TUNE_QR_THREADS, threads))
            w, q, W, V, st = E.layer_modes(conv, np.zeros(P, int), kx, ky, precision=form)
        finally:
            _lib.check(lib.wb_set_tuning(_lib.WB_TUNE_QR_THREADS, 0))
        assert not (st.cpu().numpy() & ~8).any()
        w, W = w.cpu().numpy(), W.cpu().numpy()
        if ref is None:
            ref = w[0], W[0]
            om2 = O.layer_operator(kx[0], ky[0], *(conv.slot(k)[0].cpu().numpy() for k in range(3)))[0]
            # backward error of a Schur form and one triangular solve: a few n units of roundoff
            # (double-float 2^-47; the Newton-refined FP32 pairs are FP64-class to 1e-9)
            unit = {'double': 2.3e-16, 'mixed_df64': 7.2e-15, 'mixed': 1e-10}[form]
            res = np.abs(om2 @ W[0] - W[0] * w[0]).max()
            assert res <= 40 * om2.shape[0] * unit * np.abs(om2).sum(axis=1).max(), res
        for p in (0, P // 2, P - 1):
            assert np.array_equal(w[p], ref[0]) and np.array_equal(W[p], ref[1]), (P, threads, p)
