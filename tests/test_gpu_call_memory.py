"""A self-contained call gives its device memory back, but for the 64 MiB that
are kept for the next one: after calls that took 1.3 GB, one alone and several
at once, the device has as much free memory as after a small call, within that
and the driver's own 32 MiB blocks."""
import ctypes as C
import threading

import numpy as np
import pytest

from texo_gb300.placer import routing_demand

pytestmark = pytest.mark.gpu


def free_bytes():
    free, total = C.c_size_t(), C.c_size_t()
    assert C.CDLL("libcuda.so.1").cuMemGetInfo_v2(C.byref(free), C.byref(total)) == 0
    return free.value


def test_memory_of_large_calls_is_given_back():
    box = np.array([[1.0, 5.0, 2.0, 9.0]])
    routing_demand(40, 40, box)
    before = free_bytes()
    routing_demand(6400, 6400, box)   # 2 x 6401^2 + 2 x 6400^2 words
    assert before - free_bytes() <= (64 + 32) << 20
    threads = [threading.Thread(target=routing_demand, args=(1600, 1600, box)) for _ in range(8)]   # 82 MB each
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert before - free_bytes() <= (64 + 32) << 20
