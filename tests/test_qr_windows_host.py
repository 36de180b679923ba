"""The windowed QR sweep (wavebit_gb300/csrc/wb_qr.cuh) restated in NumPy: which warp touches which
element of H and Z in which tick. Held to the element-by-element sweep bit for bit, whichever of the
tick's concurrent parts (the far update of the window before; the chase and its near columns) runs
first, with their reads and writes checked for overlap and every index for its range."""
import numpy as np
import pytest


class Mat:
    def __init__(self, a):
        self.a, self.read, self.written = a, set(), set()

    def get(self, i, j):
        assert 0 <= i < len(self.a) and 0 <= j < len(self.a)
        self.read.add((i, j))
        return self.a[i, j]

    def put(self, i, j, v):
        assert 0 <= i < len(self.a) and 0 <= j < len(self.a)
        self.written.add((i, j))
        self.a[i, j] = v


def reflector(alpha, x):
    if x == 0 and alpha.imag == 0:
        return 0j, 0j, 0.0, alpha.real, True
    beta = -np.copysign(np.sqrt(abs(alpha) ** 2 + x * x), alpha.real)
    return (beta - alpha) / beta, x / (alpha - beta), -(x / beta), beta, False


def left(ref, a, b):
    s = np.conj(ref[0]) * a + b * ref[2]
    return a - s, b - s * ref[1]


def right(ref, a, b):
    s = ref[0] * a + b * ref[2]
    return a - s, b - s * np.conj(ref[1])


def shift(h, i):
    t, u = h(i, i), np.sqrt(h(i - 1, i)) * np.sqrt(h(i, i - 1))
    if u == 0:
        return t
    x = (h(i - 1, i - 1) - t) * 0.5
    y = np.sqrt(x * x + u * u)
    if (np.conj(x) * y).real < 0:
        y = -y
    return t - u * (u / (x + y))


def block(h, i):
    for k in range(i, 0, -1):
        if abs(h(k, k - 1)) <= 1e-14 * (abs(h(k, k)) + abs(h(k - 1, k - 1))):
            return k
    return 0


def make_real(sd):
    if sd.imag == 0:
        return sd, 1.0, False
    return complex(abs(sd)), sd * (1 / abs(sd)), True


def by_element(H, Z):
    n, i = len(H), len(H) - 1
    h = lambda r, c: H[r, c]  # noqa: E731
    while i >= 0:
        lo = block(h, i)
        if lo >= i:
            i -= 1
            continue
        if lo > 0:
            H[lo, lo - 1] = 0
        ref = reflector(H[lo, lo] - shift(h, i), H[lo + 1, lo].real)
        for k in range(lo, i):
            for c in range(k, n):
                H[k, c], H[k + 1, c] = left(ref, H[k, c], H[k + 1, c])
            for r in range(min(k + 2, i) + 1):
                H[r, k], H[r, k + 1] = right(ref, H[r, k], H[r, k + 1])
            for r in range(n):
                Z[r, k], Z[r, k + 1] = right(ref, Z[r, k], Z[r, k + 1])
            if k + 1 < i:
                ref = reflector(H[k + 1, k], H[k + 2, k].real)
                if not ref[4]:
                    H[k + 1, k] = ref[3]
                H[k + 2, k] = 0
        H[i, i - 1], sc, scaled = make_real(H[i, i - 1])
        if scaled:
            for c in range(i + 1, n):
                H[i, c] = np.conj(sc) * H[i, c]
            for r in range(i):
                H[r, i] = sc * H[r, i]
            for r in range(n):
                Z[r, i] = sc * Z[r, i]


class Windowed:
    def __init__(self, H, Z, m, far_first):
        self.H, self.Z, self.n, self.m, self.far_first = Mat(H), Mat(Z), len(H), m, far_first
        self.ld = 3 * m + 5
        self.tiles = [np.full((m, self.ld), np.nan + 0j) for _ in range(2)]
        self.i, self.k0, self.kp, self.base, self.cur, self.drain = self.n - 1, -1, 0, 0, 0, 1 << 30
        self.idle = 0

    def decide(self):
        h = self.H.get
        if self.k0 < 0:
            while True:
                if self.i < 0:
                    return 'done'
                lo = block(h, self.i)
                if lo < self.i:
                    break
                self.i -= 1
            if lo > 0:
                self.H.put(lo, lo - 1, 0)
            if min(lo + 2 * self.m + 1, self.i) >= self.drain:
                self.drain = 1 << 30
                self.idle += 1
                return 'idle'
            i = self.i
            self.core = [h(lo, lo), h(lo, lo + 1), h(lo + 1, lo), h(lo + 1, lo + 1),
                         h(lo + 2, lo + 1) if lo + 2 <= i else 0j]
            self.above = (h(lo - 1, lo), h(lo - 1, lo + 1)) if lo > 0 else (0j, 0j)
            self.ref = reflector(self.core[0] - shift(h, i), self.core[2].real)
            self.k0 = self.kp = self.base = lo
        self.drain = 1 << 30
        return 'window'

    def load(self, tile, c0, cmax, base, e):
        tile[:] = np.nan
        nrow = e + 3 - base
        assert nrow <= self.ld
        for j, c in enumerate(range(c0, min(cmax, c0 + self.m - 1) + 1)):
            for r in range(nrow):
                tile[j, r] = self.H.get(base + r, c) if base + r <= min(c + 1, self.i) else 0

    def chase(self, before):
        H, m, i, k0 = self.H, self.m, self.i, self.k0
        k1 = min(k0 + m, i)
        cmax, tile, last = min(k1 + 1, i), self.tiles[self.cur], k1 == i
        if self.kp == k0:
            self.load(tile, k0 + 2, cmax, self.base, k1)
        o = k0 - self.base
        lanes = [j for j in range(m) if k0 + 2 + j <= cmax]
        a = {j: tile[j, o] for j in lanes}
        b = {j: tile[j, o + 1] for j in lanes}
        refs, sc, scaled = [], 1.0, False
        c00, c01, c10, c11, c21 = self.core
        x, y = self.above
        ref = self.ref
        for k in range(k0, k1):
            q = k - k0
            refs.append(ref)
            p22, p32, yn, cn = 0j, 0j, 0j, 0j
            if k + 2 <= i:
                p22, p32 = tile[q, o + q + 2], tile[q, o + q + 3]
                assert not np.isnan(p22) and not np.isnan(p32)
            for j in lanes:
                an, bn = left(ref, a[j], b[j])
                if j == q:
                    yn, cn = an, bn
                elif j > q:
                    H.put(k, k0 + 2 + j, an)
                a[j], b[j] = bn, tile[j, o + q + 2]
            h00, h10 = left(ref, c00, c10)
            h01, h11 = left(ref, c01, c11)
            h00, h01 = right(ref, h00, h01)
            h10, h11 = right(ref, h10, h11)
            s = c21 * ref[2]
            h20, h21 = -s, c21 - s * np.conj(ref[1])
            xf, yf = right(ref, x, y)
            sub = h10
            if k + 1 < i:
                ref = reflector(h10, h20.real)
                if not ref[4]:
                    sub = ref[3]
                c00, c10, c01, c11, c21, x, y = h11, h21, cn, p22, p32, h01, yn
            else:
                sub, sc, scaled = make_real(h10)
                if scaled:
                    h01, yf = sc * h01, sc * yf
                H.put(k, k + 1, h01)
                H.put(k + 1, k + 1, h11)
            H.put(k, k, h00)
            H.put(k + 1, k, sub)
            if k > 0:
                H.put(k - 1, k, xf)
                H.put(k - 1, k + 1, yf)
        k2 = min(k1 + m, i)
        if not last:                                # the near columns: those of the window after
            near, kp, top = self.tiles[self.cur ^ 1], self.kp, min(k2 + 1, i)
            self.load(near, k1 + 2, top, kp, k2)
            for j, c in enumerate(range(k1 + 2, top + 1)):
                v = near[j, 0]
                for r, rf in enumerate((before['refs'] if k0 > kp else []) + refs):
                    w, v = left(rf, v, near[j, r + 1])
                    H.put(kp + r, c, w)
                near[j, k1 - kp] = v
        self.core, self.above, self.ref = [c00, c01, c10, c11, c21], (x, y), ref
        if last:
            self.drain, self.k0 = k0, -1
        else:
            self.base, self.kp, self.k0, self.cur = self.kp, k0, k1, self.cur ^ 1
        return dict(k0=k0, k1=k1, refs=refs, sc=sc, scaled=scaled, cfar=min(min(k2 + m, i) + 1, i) + 1)

    def far(self, g):
        if g is None:
            return
        k0, k1 = g['k0'], g['k1']
        for c in range(g['cfar'], self.n):
            a = self.H.get(k0, c)
            for q, rf in enumerate(g['refs']):
                w, a = left(rf, a, self.H.get(k0 + q + 1, c))
                self.H.put(k0 + q, c, w)
            self.H.put(k1, c, np.conj(g['sc']) * a if g['scaled'] else a)
        for M, rows, gap in ((self.H, max(0, k1 - 2), 2), (self.Z, self.n, -self.n)):
            for r in range(rows):
                kst = max(k0, r + gap)
                if kst >= k1:
                    continue
                a = M.get(r, kst)
                for k in range(kst, k1):
                    w, a = right(g['refs'][k - k0], a, M.get(r, k + 1))
                    M.put(r, k, w)
                M.put(r, k1, g['sc'] * a if g['scaled'] else a)

    def run(self):
        before = None
        while True:
            H = self.H
            H.read.clear(), H.written.clear()
            if self.far_first:
                self.far(before)
            fr, fw = set(H.read), set(H.written)
            H.read.clear(), H.written.clear()
            kind = self.decide()
            now = self.chase(before) if kind == 'window' else None
            if self.far_first:
                assert not fw & (H.read | H.written) and not fr & H.written
            else:
                self.far(before)
            before = now
            if kind == 'done':
                return


@pytest.mark.parametrize('n', [1, 2, 3, 8, 17, 34])
@pytest.mark.parametrize('m', [2, 3, 8, 16])
@pytest.mark.parametrize('far_first', [True, False])
def test_windows_equal_the_sweep_by_elements(n, m, far_first):
    rng = np.random.default_rng(100 * n + m)
    A = np.triu(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), -1)
    for k in range(1, n):
        A[k, k - 1] = abs(A[k, k - 1])
    if n > 8:
        A[n // 2, n // 2 - 1] = 0                   # a block that splits
    H1, Z1, H2, Z2 = A.copy(), np.eye(n, dtype=complex), A.copy(), np.eye(n, dtype=complex)
    by_element(H1, Z1)
    Windowed(H2, Z2, m, far_first).run()
    assert np.array_equal(np.triu(H1), np.triu(H2)) and np.array_equal(Z1, Z2)
    assert np.abs(Z2 @ np.triu(H2) @ Z2.conj().T - A).max() < 1e-12
