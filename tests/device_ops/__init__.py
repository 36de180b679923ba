"""Builds tests/device_ops/ops.cu against the library and binds it."""
import ctypes
import os
import shutil
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(os.path.dirname(HERE)), 'wavebit_gb300')
_ops = None


def load():
    """The bound library (built once a process)."""
    global _ops
    if _ops is None:
        from wavebit_gb300 import _lib
        _lib.load()
        out = os.path.join(tempfile.mkdtemp(prefix='device_ops'), 'libops.so')
        nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
        subprocess.run([nvcc, '-gencode', 'arch=compute_103a,code=sm_103a', '-O2', '-std=c++17', '-shared', '-Xcompiler',
                        '-fPIC', '--expt-relaxed-constexpr', '-I', os.path.join(PKG, 'csrc'), '-o', out,
                        os.path.join(HERE, 'ops.cu'), '-L', PKG, '-l:libwbgpu.so', '-Xlinker', f'-rpath={PKG}'],
                       check=True, capture_output=True)
        _ops = ctypes.CDLL(out)
        i, ll, p, d = ctypes.c_int, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_double
        _ops.ops_getrf.argtypes = [i, i, i, p, ll, p, p]
        _ops.ops_getrs.argtypes = [i, i, i, p, ll, p, p, i, i]
        _ops.ops_zgemm.argtypes = [i, i, i, i, d, d, p, p, p, i, p, p, i, d, d, p, p]
        _ops.ops_schur.argtypes = [i, i, p, p, p, p, p]
        _ops.ops_rsqrt.argtypes = [i, p, p, p, p]
    return _ops
