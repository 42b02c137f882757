"""The demand map of boxes whose pieces end at the fabric's edges, on tile
centres and borders, without a run of whole tiles between their edges, without
extent, and outside: against the oracle's FP64 sums to 1e-11 (at most a few
dozen rectangles a tile, each rounded to 2^-41)."""
import numpy as np
import pytest

from oracle import ffi
from texo_gb300.placer import routing_demand


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(1, 1), (2, 3), (33, 7), (64, 31)])
def test_boxes_at_the_edges(W, H):
    marks = sorted({-3.0, -0.75, -0.5, -0.25, 0.0, 0.5, 1.0, 1.25, W / 2, W - 1.5, W - 1.0, W - 0.5, W - 0.25, W + 2.5})
    marks_y = sorted({-2.0, -0.5, 0.0, 0.3, 0.5, H - 1.0, H - 0.5, H + 0.0, H + 4.0})
    boxes = [(a, b, c, d) for i, a in enumerate(marks) for b in marks[i:] for k, c in enumerate(marks_y)
             for d in marks_y[k::3]]
    for part in np.array_split(np.array(boxes), 40):
        h, v, _ = routing_demand(W, H, part)
        rh, rv = ffi.routing_demand(W, H, part)[:2]
        assert np.max(np.abs(h - np.asarray(rh).reshape(H, W))) <= 1e-11
        assert np.max(np.abs(v - np.asarray(rv).reshape(H, W))) <= 1e-11
