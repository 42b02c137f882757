"""A box whose width is beyond FP64 has no demand that is a number; the tiles
that it does not touch have none, and other boxes' demand there is unchanged."""
import numpy as np
import pytest

from texo_gb300.placer import routing_demand


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi", [(3.0, 5.0), (3.0, 3.0), (3.5, 4.25), (0.0, 1.0), (11.0, 11.0)])
def test_tiles_beside_a_box_of_infinite_width(lo, hi):
    H = 12
    wide = 1.7e308
    touched = np.array([min(y + 0.5, hi + 0.5) - max(y - 0.5, lo - 0.5) > 0 for y in range(H)])
    other = [2.0, 4.5, 0.25, 11.0]
    alone_h, alone_v, _ = routing_demand(9, H, np.array([other]))
    h, v, _ = routing_demand(9, H, np.array([[-wide, wide, lo, hi], other]))
    assert np.array_equal(h[~touched], alone_h[~touched]) and np.array_equal(v[~touched], alone_v[~touched])
    h, v, _ = routing_demand(H, 9, np.array([[lo, hi, -wide, wide]]))
    assert not h[:, ~touched].any() and not v[:, ~touched].any()
