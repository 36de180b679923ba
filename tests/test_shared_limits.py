"""A kernel's limit of dynamic shared memory is one constant, set through allow_shared: set to the size of the call
at hand, one host thread's smaller call lowers it between another's setting and launch, which then fails."""
import glob
import os
import re
import threading

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'wavebit_gb300', 'csrc')


def _sources():
    return {os.path.basename(f): re.sub(r'//[^\n]*', '', open(f).read())
            for pat in ('*.cu', '*.cuh', '*.h') for f in glob.glob(os.path.join(CSRC, pat))}


def test_limits_are_constants():
    calls = 0
    for name, text in _sources().items():
        if name == 'wb_kernels.h':
            continue
        assert 'cudaFuncAttributeMaxDynamicSharedMemorySize' not in text, name
        consts = set(re.findall(r'constexpr (?:int|size_t) (\w+)', text)) | {'kVectorShared'}
        for call in re.finditer(r'allow_shared\(([^;]*?), ((?:\(int\))?[\w:]+(?: [*/] \w+)*)\)', text):
            words = [w.split('::')[-1] for w in re.findall(r'[A-Za-z_][\w:]*', call.group(2)) if w != 'int']
            assert all(w in consts or w in ('kSmem', 'kSmemBytes', 'most') for w in words), (name, call.group(0))
            calls += 1
        calls -= text.count('allow_shared(')
    assert calls == 0                                                 # every call was read


def test_a_launch_with_vectors_in_shared_memory_has_a_limit():
    """Kernels launched with dynamic shared memory that grows with n: past 48 KB they need their limit raised"""
    text = _sources()['wb_eig.cu'] + _sources()['wb_linalg.cu'] + _sources()['wb_solve.cu']
    for kernel, size in re.findall(r'(\w+)<?R?>?<<<[^;]*?, \d*\w*, ([^;]*?), s>>>', text):
        if size.strip() == '0':
            continue
        assert re.search(r'allow_shared\((?:tri::)?' + kernel, text) or kernel in ('kernel', 'trsm_upper_f32_kernel'), kernel


@pytest.mark.gpu
def test_threads_with_calls_of_their_own_sizes():
    torch = pytest.importorskip('torch')
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from wavebit_gb300 import _lib, engine as E
    rng = np.random.default_rng(0)
    cases = []
    for hu, P in ((8, 40), (31, 3), (63, 2)):                          # n = 34, 126, 254
        eps = np.where(rng.random((1, 1, 300)) < 0.5, 1.0, 6.0).astype(complex)
        kx = np.tile(np.arange(-hu, hu + 1) * 0.71 + 0.13, (P, 1))
        conv = E.assemble(torch.as_tensor(eps, device='cuda'), hu, 0)
        cases.append((conv, np.zeros(P, int), kx, np.full((P, 2 * hu + 1), 0.21)))
    want = [[E.layer_modes(*c, precision=p)[0].cpu().numpy() for p in ('double', 'mixed')] for c in cases]
    torch.cuda.synchronize()
    failed = []

    def work(k):
        try:
            h = _lib.Handle(0, 2 << 30)
            with torch.cuda.stream(torch.cuda.Stream()):
                for t in range(12):
                    w = E.layer_modes(*cases[k], precision=('double', 'mixed')[t % 2], handle=h)[0]
                    w, ref = w.cpu().numpy(), want[k][t % 2]
                    if not np.abs(w - ref).max() <= (1e-8 if t % 2 else 0.0) * np.abs(ref).max():
                        failed.append((k, t, 'other eigenvalues'))
            torch.cuda.synchronize()
            h.close()
        except Exception as e:                                        # noqa: BLE001
            failed.append((k, repr(e)))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    [t.start() for t in threads]
    [t.join(120) for t in threads]
    assert not failed, failed
