"""The first register-clustering calls of a process, of several threads at
once: every one computes with a complete window table. Areas equal those of a
later call bit for bit, and the oracle's to 1e-12, as the other cases."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import threading
import numpy as np
from oracle import ffi
from texo_gb300 import routability
rng = np.random.default_rng(7)
n = 300
xy = rng.uniform(0, 9, (n, 2))
cl = np.stack([rng.integers(0, 2, n), np.zeros(n, np.int64)], axis=1)
ce = rng.integers(0, 5, n)
start = threading.Barrier(8)
got = [None] * 8

def run(k):
    start.wait()
    got[k] = routability.register_clustering_areas(xy, cl, ce, 9000)[0]

threads = [threading.Thread(target=run, args=(k,)) for k in range(8)]
for t in threads:
    t.start()
for t in threads:
    t.join()
later, _ = routability.register_clustering_areas(xy, cl, ce, 9000)
assert all(np.array_equal(g, later) for g in got)
code, expected = ffi.register_clustering_areas(xy, cl, ce, 9000)
assert code == 0 and np.max(np.abs(later - expected) / expected) <= 1e-12
"""


def test_the_first_calls_of_several_threads():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", CODE], cwd=root, check=True, timeout=300)
