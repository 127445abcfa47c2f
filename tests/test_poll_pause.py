"""CPU: the wait loops' pause gives the core away where another thread wants it,
and then sleeps between its looks (at least 10 us, so that a wait of 0.2 ms
has 20 at most); the thread's timer slack is put back."""
import ctypes as C
import os
import threading
import time

from compute_vp9_b200 import cuda_lib

PR_GET_TIMERSLACK = 30


def _pause():
    pause = cuda_lib().cvp9_poll_pause
    pause.argtypes, pause.restype = [C.POINTER(C.c_uint), C.c_double], None
    return pause


def test_sleeps_where_told_and_after_long_waits():
    pause, naps = _pause(), C.c_uint(10 ** 6)
    prctl = C.CDLL(None).prctl
    slack = prctl(PR_GET_TIMERSLACK, 0, 0, 0, 0)
    looks = 0
    for _ in range(200):                       # waits of 0.2 ms
        t0 = now = time.monotonic()
        while now - t0 < 200e-6:
            pause(naps, now - t0)
            now = time.monotonic()
            looks += 1
    assert 200 <= looks <= 200 * 20
    naps.value = 0
    t0 = time.monotonic()
    pause(naps, 1e-3)
    assert time.monotonic() - t0 >= 20e-6 and naps.value == 0
    assert prctl(PR_GET_TIMERSLACK, 0, 0, 0, 0) == slack


def test_notices_another_thread_on_its_core():
    pause, naps, stop = _pause(), C.c_uint(0), threading.Event()
    cores = os.sched_getaffinity(0)
    os.sched_setaffinity(0, {min(cores)})      # the new thread inherits it
    try:
        def busy():
            while not stop.is_set():
                sum(range(1000))
        t = threading.Thread(target=busy)
        t.start()
        end = time.monotonic() + 10
        while not naps.value and time.monotonic() < end:
            pause(naps, 0.0)
        stop.set()
        t.join()
    finally:
        os.sched_setaffinity(0, cores)
    assert naps.value > 0
