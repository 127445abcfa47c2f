"""A superblock whose neighbour is slow waits for at least half a second before
the frame reports CVP9_JOB_TIMEOUT (the limit that it has had), and gives up
within a few seconds."""
import ctypes as C

import pytest

from compute_vp9_b200 import CVP9_OK, cuda_lib

pytestmark = pytest.mark.gpu

JOB_TIMEOUT = 1 << 2


def test_neighbour_wait_length():
    lib = cuda_lib()
    lib.cuda_backend_selftest_wait_limit.argtypes = [C.c_int, C.POINTER(C.c_uint32), C.POINTER(C.c_float)]
    status, ms = C.c_uint32(), C.c_float()
    assert lib.cuda_backend_selftest_wait_limit(-1, C.byref(status), C.byref(ms)) == CVP9_OK
    assert status.value & JOB_TIMEOUT
    assert 500.0 < ms.value < 5000.0, ms.value
