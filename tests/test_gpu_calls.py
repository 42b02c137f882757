"""Self-contained calls share kept streams and a memory pool, and the register
clustering orders its control sets by digits of the keys.

The calls of many threads (more than there are kept streams) give each the
result of the call alone, bit for bit. Keys that together need more than 64
bits are ordered one key after the other: relabelling the control sets in an
order-preserving way changes no area at all, and the areas are the oracle's to
1e-12 relative (sums of a few thousand terms of at most 1, each within 1e-15)."""
import threading

import numpy as np
import pytest

from oracle import ffi
from texo_gb300 import routability
from texo_gb300.placer import quadratic_solve, routing_demand

pytestmark = pytest.mark.gpu


def test_calls_of_many_threads_do_not_mix():
    rng = np.random.default_rng(4)
    corners = np.sort(rng.uniform(0, 39, (12, 500, 2, 2)), axis=2)
    boxes = [np.stack([c[:, 0, 0], c[:, 1, 0], c[:, 0, 1], c[:, 1, 1]], axis=1) for c in corners]
    ptr = np.arange(0, 129, 2)
    idx = np.stack([(np.arange(64) + 1) % 64, (np.arange(64) - 1) % 64], axis=1).reshape(-1)
    rhs = rng.normal(size=(12, 64))

    def work(k):
        h, v, _ = routing_demand(40, 40, boxes[k])
        x, _ = quadratic_solve(np.full(64, 3.0), ptr, idx, np.ones(128), rhs[k])
        return h, v, x

    alone = [work(k) for k in range(12)]
    got = [None] * 12

    def run(k):
        got[k] = [work(k) for _ in range(5)]

    threads = [threading.Thread(target=run, args=(k,)) for k in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(12):
        for r in got[k]:
            assert all(np.array_equal(a, b) for a, b in zip(r, alone[k]))


@pytest.mark.parametrize("n,sets,enables", [(1, 1, 1), (31, 2, 3), (600, 5, 7), (4100, 1, 40)])
def test_wide_keys_order_as_narrow_ones(n, sets, enables):
    rng = np.random.default_rng(n)
    xy = rng.uniform(0, 30, (n, 2))
    clock, lsr, ce = rng.integers(0, sets, n), rng.integers(0, 2, n), rng.integers(0, enables, n)

    def widen(v):   # order-preserving, all 64 bits in use
        labels = np.sort(rng.integers(0, 2**63, v.max() + 1).astype(np.uint64) * np.uint64(2))
        labels[0], labels[-1] = 0, 2**64 - 1
        return labels[v]

    narrow, _ = routability.register_clustering_areas(xy, np.stack([clock, lsr], axis=1), ce, 9000)
    wide, _ = routability.register_clustering_areas(xy, np.stack([widen(clock), widen(lsr)], axis=1), widen(ce), 9000)
    assert np.array_equal(narrow, wide)
    code, expected = ffi.register_clustering_areas(xy, np.stack([clock, lsr], axis=1), ce, 9000)
    assert code == 0
    assert np.max(np.abs(narrow - expected) / expected) <= 1e-12
