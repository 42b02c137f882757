"""The auction where one block runs the rounds alone (at most 64 bidders), and
where walks leave the table of the diamond's points (1024 of them, rings to
22): bidders of the lone block's limit less or more one on one tile, and free
BELs only beyond ring 22, with one BEL a tile and with several. Whole numbers:
the oracle's restatement of the parallel rounds gives the same assignment,
prices, rounds and bids."""
import numpy as np
import pytest

from oracle import ffi
from texo_gb300 import legalize


@pytest.mark.gpu
@pytest.mark.parametrize("bidders", [1, 63, 64, 65, 129])
@pytest.mark.parametrize("side,cap,free_from", [(30, 1, 0), (30, 3, 0), (70, 1, 22), (70, 2, 30)])
def test_bit_exact_against_the_parallel_restatement(bidders, side, cap, free_from):
    tiles = np.abs(np.arange(side)[:, None] - 3) + np.abs(np.arange(side)[None, :] - 5)
    capacity = np.full((1, side, side), cap, dtype=np.int64)
    occupied = np.repeat((tiles < free_from).reshape(-1), cap).astype(np.uint8)
    grid = legalize.site_grid(capacity, occupied=occupied)
    kind = np.zeros(bidders, np.uint32)
    target = np.tile(np.array([5, 3], np.uint32), (bidders, 1))
    target[1::3, 0] += 1
    r = legalize.auction_singletons(grid, kind, target, cost_scale=2)
    code, a, prices, st = ffi.auction_singletons(grid, kind, target, cost_scale=2, jacobi=True)
    assert code == 0
    assert np.array_equal(r.assignment, a) and np.array_equal(r.prices.astype(np.uint64), prices)
    assert (r.stats["rounds"], r.stats["bids"]) == (st["rounds"], st["bids"])
    assert (r.stats["unmatched"], r.stats["total_base_cost"]) == (st["unmatched"], st["total_base_cost"])
