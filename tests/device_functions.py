"""The kernels of device_functions.cu, built with nvcc on first use."""
import ctypes
import os
import subprocess
import tempfile

from yastn_gb300 import build

_lib = []


def lib():
    if not _lib:
        src = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'device_functions.cu')
        so = os.path.join(tempfile.mkdtemp(), 'device_functions.so')
        subprocess.run([build.nvcc()] + build.ARCH + build.FLAGS + ['-shared', src, '-o', so], check=True)
        _lib.append(ctypes.CDLL(so))
    return _lib[0]
