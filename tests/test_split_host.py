"""Two rules of the mixed form's kernels restated in NumPy: an FP64 number as two floats by integer
operations (dd_split, wavebit_gb300/csrc/wb_linalg.cu) against the conversions it replaces, and the
FP32 test by which group_link_kernel (wavebit_gb300/csrc/wb_solve.cu) passes a coupling over."""
import numpy as np
import pytest


def _split(x):
    b = x.view(np.uint64)
    h, l = (b >> np.uint64(32)).astype(np.int64), (b & np.uint64(0xffffffff)).astype(np.int64)
    e = (h >> 20) & 0x7ff
    sign = h & 0x80000000
    top = ((h & 0xfffff) << 3) | (l >> 29)
    low = l & 0x1fffffff
    up = (low + (top & 1) > 0x10000000).astype(np.int64)
    hi = (sign | ((((e - 896) << 23) | top) + up)).astype(np.uint32).view(np.float32)
    rem = low - (up << 29)
    rem = np.where(sign != 0, -rem, rem).astype(np.int32).astype(np.float32)
    scale = ((e - 1075 + 127) << 23).astype(np.uint32).view(np.float32)
    return hi, rem * scale


@pytest.mark.parametrize('exponent', [960, 961, 1000, 1022, 1023, 1024, 1100, 1139, 1140])
def test_split_is_the_conversions(exponent):
    rng = np.random.default_rng(exponent)
    m = rng.integers(0, 1 << 52, 200000, dtype=np.uint64)
    k = rng.integers(0, 53, m.size, dtype=np.uint64)
    m[::3] &= ~((np.uint64(1) << k[::3]) - np.uint64(1))          # short mantissas
    m[1::5] = (m[1::5] & ~np.uint64(0x1fffffff)) | np.uint64(0x10000000)   # ties
    m[:4] = [0, (1 << 52) - 1, 0x10000000, 0x30000000]
    s = rng.integers(0, 2, m.size, dtype=np.uint64) << np.uint64(63)
    x = (s | (np.uint64(exponent) << np.uint64(52)) | m).view(np.float64)
    hi = x.astype(np.float32)
    lo = (x - hi.astype(np.float64)).astype(np.float32)
    got_hi, got_lo = _split(x)
    assert np.array_equal(got_hi.view(np.uint32), hi.view(np.uint32))
    assert np.array_equal(got_lo.view(np.uint32), lo.view(np.uint32))


def test_a_coupling_passed_over_is_weak():
    couple = 0.02
    rng = np.random.default_rng(0)
    n = 400000
    g = (rng.standard_normal((2, n)) * 10.0 ** rng.uniform(-40, 20, n)).astype(np.float32)
    ratio = 10.0 ** rng.uniform(-2, 2, n)
    ratio[::2] = 1.0 + rng.uniform(-1e-3, 1e-3, n // 2)           # at the threshold
    angle = rng.uniform(0, 2 * np.pi, n)
    angle[::4] = np.pi / 4
    g[1, 1::4] = g[0, 1::4]
    mod = np.hypot(g[0].astype(float), g[1].astype(float))
    gap = mod / couple * ratio
    d = np.array([gap * np.cos(angle), gap * np.sin(angle)])
    gm = np.abs(g).max(axis=0)
    with np.errstate(over='ignore', under='ignore'):
        dm = np.abs(d.astype(np.float32)).max(axis=0)
        skip = (gm * np.float32(1.41422) <= np.float32(couple) * np.float32(0.9999) * dm) & (dm > 1e-30) & (gm < 1e30)
    assert skip.any() and not (skip & (mod > couple * np.hypot(d[0], d[1]))).any()
