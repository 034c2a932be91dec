"""The QR's waits after one has run out: the first one takes its whole limit (a few seconds), the
others return at once, so that a failed factorisation of a few hundred panels ends in seconds."""
import ctypes
import time

import pytest

import device_functions

pytestmark = pytest.mark.gpu


def test_one_timeout_ends_all_waits(cuda_device):
    import torch
    words = torch.zeros(2, dtype=torch.int64, device='cuda')  # the flag, the error word
    lib = device_functions.lib()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    st = lib.t_qr_waits(ctypes.c_void_p(words.data_ptr()), ctypes.c_void_p(words.data_ptr() + 8), 200,
                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    took = time.perf_counter() - t0
    assert st == 0 and words.tolist() == [0, 1]
    assert took < 30.0, took
