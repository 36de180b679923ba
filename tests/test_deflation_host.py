"""The FP64 sweep's rule for pairs that cannot be told apart (same_pair, wavebit_gb300/csrc/wb_qr.cuh), compiled for
the host: what it deflates changes neither eigenvalue of the pair by more than the rounding of their sum, and a pair that
only the small-subdiagonal test would take (a graded one) stays."""
import ctypes
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'wavebit_gb300', 'csrc')
ULP = 2.0 ** -52


@pytest.fixture(scope='module')
def rule(tmp_path_factory):
    text = open(os.path.join(CSRC, 'wb_qr.cuh')).read()
    body = re.search(r'bool same_pair\(.*?\n}', text, re.S).group(0)
    gxx = shutil.which('g++')
    if gxx is None:
        pytest.skip('g++ is not available')
    d = tmp_path_factory.mktemp('deflation')
    (d / 'r.cpp').write_text('#include <cmath>\ntemplate <class R> struct Cx { R x, y; };\n'
                             'template <class R> R cxabs1(Cx<R> a) { return std::fabs(a.x) + std::fabs(a.y); }\n'
                             'template <class R> ' + body + '\nextern "C" int rule(const double* v, double tol) {\n'
                             '  return same_pair<double>({v[0], v[1]}, {v[2], v[3]}, {v[4], v[5]}, tol); }\n')
    so = str(d / 'r.so')
    subprocess.run([gxx, '-O1', '-std=c++17', '-shared', '-fPIC', '-o', so, str(d / 'r.cpp')], check=True, capture_output=True)
    fn = ctypes.CDLL(so).rule
    fn.argtypes = [ctypes.c_void_p, ctypes.c_double]

    def call(p, t, sub, sup):
        tol = ULP * (abs(p.real) + abs(p.imag) + abs(t.real) + abs(t.imag))
        v = np.array([(p - t).real, (p - t).imag, sub, 0.0, sup.real, sup.imag])
        return bool(fn(v.ctypes.data, tol)), tol
    return call


def test_a_deflated_pair_keeps_its_eigenvalues(rule):
    rng = np.random.default_rng(0)
    taken = 0
    for _ in range(20000):
        t = complex(*rng.standard_normal(2)) * 10.0 ** rng.integers(-8, 8)
        p = t * (1 + ULP * complex(*rng.integers(-2, 3, 2)))
        sub = abs(t) * 10.0 ** rng.uniform(-40, -16)
        sup = complex(*rng.standard_normal(2)) * abs(t) * 10.0 ** rng.uniform(-20, 6)
        small, tol = rule(p, t, sub, sup)
        if small:
            taken += 1
            L = np.clongdouble
            x = (L(p) - L(t)) / 2
            y = np.sqrt(x * x + L(sub) * L(sup))
            m = (L(p) + L(t)) / 2
            off = min(max(abs(m + y - L(p)), abs(m - y - L(t))), max(abs(m + y - L(t)), abs(m - y - L(p))))
            assert float(off) <= 2 * tol
    assert taken > 1000


def test_graded_pairs_stay(rule):
    # |sub| within a rounding of the diagonals, but the eigenvalues move by sub sup / (p - t), far more
    for sup in (1e2, 1e4, 1e8):
        for sep in (1.0, 1e-3, 1e-8):
            assert not rule(1.0 + 0j, 1.0 + sep + 0j, 2e-16, sup + 0j)[0]
    assert not rule(1.0 + 0j, 1.0 + 0j, 2e-16, 1.0 + 0j)[0]            # a split of 1e-8: the shift resolves it
    assert rule(1.0 + 0j, 1.0 + 0j, 1e-17, 1e-17 + 0j)[0]
