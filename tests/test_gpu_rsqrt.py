"""The reciprocal root of the FP64 rotations, reflectors and pivots (rsqrt64, wb_num.cuh) over the whole normal range:
its start to 2^-21, itself to 2 units of 2^-53, and CUDA's rsqrt (within one of its last places) close by."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

pytestmark = pytest.mark.gpu


def test_reciprocal_roots_within_their_bounds():
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from device_ops import load
    rng = np.random.default_rng(0)
    bits = (rng.integers(1, 2047, 400000).astype(np.uint64) << np.uint64(52)) | rng.integers(0, 1 << 52, 400000).astype(np.uint64)
    v = bits.view(np.float64)
    edge = np.concatenate([2.0 ** np.arange(-1022, 1024), np.nextafter(2.0 ** np.arange(-1021, 1024), 0), [4 - 2.0 ** -50, np.finfo(float).max]])
    near = np.concatenate([1 + np.arange(4096) * 2.0 ** -52, 4 - np.arange(1, 4096) * 2.0 ** -51, rng.uniform(1, 4, 100000)])
    v = np.concatenate([v, edge, near])
    d = torch.as_tensor(v).cuda()
    out = [torch.zeros_like(d) for _ in range(3)]
    assert load().ops_rsqrt(v.size, d.data_ptr(), *(o.data_ptr() for o in out)) == 0
    torch.cuda.synchronize()
    start, full, cuda = (o.cpu().numpy() for o in out)
    want = 1 / np.sqrt(v.astype(np.longdouble))
    assert float(np.abs(start / want - 1).max()) <= 2.0 ** -21
    assert float(np.abs(full / want - 1).max()) <= 2 * 2.0 ** -53
    # a last place is 2 units of 2^-53 at the most
    assert (np.abs(full - cuda) <= 4 * 2.0 ** -53 * cuda).all()
