"""CPU: the wait loops' pause sleeps between two looks (for at least 10 us, so that
the core is another thread's meanwhile) and puts the thread's timer slack
back."""
import ctypes as C
import time

from compute_vp9_b200 import cuda_lib

PR_GET_TIMERSLACK = 30


def test_poll_pause():
    pause = cuda_lib().cvp9_poll_pause
    pause.argtypes, pause.restype = [C.c_double], None
    prctl = C.CDLL(None).prctl
    slack = prctl(PR_GET_TIMERSLACK, 0, 0, 0, 0)
    looks = 0
    for _ in range(200):                       # waits of 0.2 ms
        t0 = now = time.monotonic()
        while now - t0 < 200e-6:
            pause(now - t0)
            now = time.monotonic()
            looks += 1
    assert 200 <= looks <= 200 * 20
    t0 = time.monotonic()
    pause(1e-3)
    assert time.monotonic() - t0 >= 20e-6
    assert prctl(PR_GET_TIMERSLACK, 0, 0, 0, 0) == slack
