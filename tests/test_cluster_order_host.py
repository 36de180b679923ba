"""The order of shared-memory accesses between the CTAs of a cluster, on the CPU. A store into another
CTA's shared memory needs that CTA to have started, and to be through with what it stores there itself:
no kernel sends before its cluster has met. getrs_narrow_kernel (wavebit_gb300/csrc/wb_tri.cuh) is
restated phase by phase, its accesses checked for conflicts between two barriers and its answer held
to the solve's under every order of the CTAs."""
import itertools
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'wavebit_gb300', 'csrc')

SENDS = r'\b(?:put_remote|send|send32|send_record|next_reflector|chase_window)\s*(?:<\w+>)?\('
MEETS = r'\b(?:barrier_all|real_subdiagonal)\s*(?:<\w+>)?\('


def _body(text, name):
    at = re.search(r'__global__[^;{]*?\b' + name + r'\s*\(', text, re.S)
    i = text.index('{', at.end())
    depth = 0
    for j in range(i, len(text)):
        depth += {'{': 1, '}': -1}.get(text[j], 0)
        if depth == 0:
            return re.sub(r'//[^\n]*', '', text[i:j])
    raise AssertionError(name)


@pytest.mark.parametrize('source,kernel', [
    ('wb_tri.cuh', 'lu_panel_kernel'), ('wb_tri.cuh', 'getrs_narrow_kernel'), ('wb_hrd.cuh', 'gehrd64_kernel'),
    ('wb_eig.cu', 'gehrd_panel_cluster_kernel'), ('wb_qr.cuh', 'hseqr_kernel')])
def test_a_cluster_meets_before_its_first_remote_store(source, kernel):
    body = _body(open(os.path.join(CSRC, source)).read(), kernel)
    meet, send = re.search(MEETS, body), re.search(SENDS, body)
    assert send, 'no remote store found'
    assert meet and meet.start() < send.start()


class Shared:
    """One CTA's X; every access noted with the CTA that makes it."""

    def __init__(self, n):
        self.v, self.log = np.zeros(n, complex), []

    def get(self, cta, r):
        self.log.append((cta, r, False))
        return self.v[r]

    def put(self, cta, r, x):
        self.log.append((cta, r, True))
        self.v[r] = x


def _cta(rank, ctas, LU, b, X, nb, meet_first):
    """A CTA's run; a yield is a barrier of the cluster."""
    n = len(b)
    mine = X[rank]
    for r in range(n):
        mine.put(rank, r, b[r])
    if meet_first:
        yield
    blocks = -(-n // nb)
    for fwd in (True, False):
        rows = [(k * nb, min(n, (k + 1) * nb)) if fwd else (max(0, n - (k + 1) * nb), n - k * nb) for k in range(blocks)]
        for k, (i0, i1) in enumerate(rows):
            if rank == k % ctas:
                x = [mine.get(rank, r) for r in range(i0, i1)]
                order = range(i1 - i0) if fwd else range(i1 - i0 - 1, -1, -1)
                for t in order:
                    if not fwd:
                        x[t] = x[t] / LU[i0 + t, i0 + t]
                    for r in order:
                        if (r > t) == fwd and r != t:
                            x[r] = x[r] - LU[i0 + r, i0 + t] * x[t]
                for other in X:
                    for t, v in enumerate(x):
                        other.put(rank, i0 + t, v)
            yield
            for q in range(k + 1, blocks):
                if q % ctas == rank:
                    for r in range(*rows[q]):
                        acc = mine.get(rank, r)
                        for t in range(i0, i1):
                            acc = acc - LU[r, t] * mine.get(rank, t)
                        mine.put(rank, r, acc)
        yield


def _run(LU, b, ctas, nb, order, meet_first):
    """(the answer, whether two CTAs met at a place between two barriers, one of them writing)"""
    X = [Shared(len(b)) for _ in range(ctas)]
    runs = [_cta(r, ctas, LU, b, X, nb, meet_first) for r in range(ctas)]
    conflict, alive = False, True
    while alive:
        alive = False
        for r in order:
            alive |= next(runs[r], 'end') != 'end'
        for x in X:
            by = {}
            for cta, row, wrote in x.log:
                by.setdefault(row, set()).add((cta, wrote))
            conflict |= any(len({c for c, _ in s}) > 1 and any(w for _, w in s) for s in by.values())
            x.log.clear()
    return X[0].v, conflict


@pytest.mark.parametrize('n', [4, 7, 12, 17])
@pytest.mark.parametrize('ctas', [1, 2, 4])
def test_narrow_solve_has_one_answer_whatever_cta_runs_first(n, ctas):
    rng = np.random.default_rng(n)
    LU = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4 * np.eye(n)
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    want = np.linalg.solve((np.tril(LU, -1) + np.eye(n)) @ np.triu(LU), b)
    for order in itertools.permutations(range(ctas)):
        got, conflict = _run(LU, b, ctas, 4, order, True)
        assert not conflict
        # substitution of n unknowns: n units of roundoff times the condition, 1e3 at the most here
        assert np.abs(got - want).max() < n * 2.3e-16 * 1e3 * np.abs(want).max() + 1e-14
    # without the meeting the model finds the conflict
    if ctas > 1:
        assert any(_run(LU, b, ctas, 4, order, False)[1] for order in itertools.permutations(range(ctas)))


def test_the_sliced_product_leaves_at_one_barrier():
    """A flag that thread 0 sets when a wait runs out is read by every thread after the next barrier, and not set again
    before a barrier after that: set by the next chunk's wait, a late warp could read it for this chunk's and leave
    where the others stay. So two chunks in a row, and a panel's end, have flags of their own."""
    body = _body(open(os.path.join(CSRC, 'wb_oz.cuh')).read(), 'zgemm_kernel')
    reads = re.findall(r'if \(s_fail\[(\w+)\]\) \{ ok = false; break; \}', body)
    sets = re.findall(r's_fail\[(\w+)\] = 1;', body)
    assert reads == ['buf', '2'] and sorted(sets) == ['2', 'buf'] and 'const int buf = uses & 1' in body
    assert not re.search(r's_fail\b(?!\[)', body)
