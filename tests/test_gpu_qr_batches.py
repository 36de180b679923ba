"""The QR sweep's launch shapes past the sizes of one or two windows: by matrix size, batch and form a matrix gets clusters,
one CTA with the chase's scheduler shared or not, up to 16 warps, or the element-by-element sweep by 128, 256 or as many
threads as it has pairs. The same bits in every batch."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu


# (hu, hv): n = 22, 26 (double-float: element by element up to 22), 70, 126, 142 / 146 (one matrix an SM from 144 on),
# 162 (FP64 from 160 on: the chase's scheduler too), 254 / 258 (FP32 from 256 on: 16 warps), 318 / 322 (FP64 from 320 on)
@pytest.mark.parametrize('orders', [(5, 0), (6, 0), (3, 2), (31, 0), (35, 0), (36, 0), (4, 4), (63, 0), (64, 0), (79, 0), (80, 0)])
@pytest.mark.parametrize('form', ['double', 'mixed_df64', 'mixed'])
def test_bits_over_batches_and_shapes(orders, form):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from oracle import rcwa_oracle as O
    from wavebit_gb300 import engine as E
    hu, hv = orders
    rng = np.random.default_rng(hu)
    eps = np.where(rng.random((1, 1 if hv == 0 else 24, 300)) < 0.5, 1.0, 6.0).astype(complex)
    conv = E.assemble(torch.as_tensor(eps, device='cuda'), hu, hv)
    u, v = np.arange(-hu, hu + 1) * 0.71, np.arange(-hv, hv + 1) * 0.83
    n = 2 * len(u) * len(v)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ref = None
    batches = (1, sms // 2 + 4, sms, sms + 8) + ((4 * sms + 2,) if n <= 70 else (2 * sms + 8,) if n < 200 else ())
    for P in batches:
        kx = torch.as_tensor(np.tile(u + 0.13, 2 * hv + 1), device='cuda').expand(P, n // 2).contiguous()
        ky = torch.as_tensor(np.repeat(v + 0.21, 2 * hu + 1), device='cuda').expand(P, n // 2).contiguous()
        pl = torch.zeros(P, dtype=torch.int32, device='cuda')
        w, q, W, V, st = E.layer_modes(conv, pl, kx, ky, precision=form)
        assert not (st.cpu().numpy() & ~8).any()
        if ref is None:
            ref = w[0].clone(), W[0].clone()
            w0, W0 = w[0].cpu().numpy(), W[0].cpu().numpy()
            om2 = O.layer_operator(kx[0].cpu().numpy(), ky[0].cpu().numpy(), *(conv.slot(k)[0].cpu().numpy() for k in range(3)))[0]
            # backward error of a Schur form and one triangular solve: a few n units of roundoff (double-float 2^-47;
            # the Newton-refined FP32 pairs are FP64-class to 1e-9)
            unit = {'double': 2.3e-16, 'mixed_df64': 7.2e-15, 'mixed': 1e-10}[form]
            assert np.abs(om2 @ W0 - W0 * w0).max() <= 40 * n * unit * np.abs(om2).sum(axis=1).max()
        if form == 'mixed':        # its Hessenberg panel's norms follow the threads a batch gets: other last bits
            lim = 1e-9 * ref[0].abs().max()
            assert all((w[p] - ref[0]).abs().max() <= lim for p in (0, P // 2, P - 1)), P
        else:
            assert all(torch.equal(w[p], ref[0]) and torch.equal(W[p], ref[1]) for p in (0, P // 2, P - 1)), P
