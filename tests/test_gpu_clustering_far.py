"""Registers so far out that the window's edges x - w and x + w are one FP64
number have no expectation and are refused, as the oracle refuses them; those
just inside are accepted by both."""
import numpy as np
import pytest

from oracle import ffi
from texo_gb300 import abi, routability

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e12, 2.0**53, 2.0**54, 2.0**56, 1e17, -1e17, 1e30, 1e39, 1e300])
@pytest.mark.parametrize("axis", [0, 1])
def test_far_registers_are_refused_as_the_oracle_refuses_them(far, axis):
    xy = np.array([[3.0, 4.0], [3.5, 4.0], [5.0, 2.0]])
    xy[1, axis] = far
    cl, ce = np.zeros((3, 2), np.uint64), np.array([1, 2, 1], np.uint64)
    w = 2.5 * np.sqrt(1e-5 * 40000)
    code, expected = ffi.register_clustering_areas(xy, cl, ce, 40000)
    assert (code != 0) == (far + w == far - w)
    if code:
        with pytest.raises(abi.TexoGpError) as e:
            routability.register_clustering_areas(xy, cl, ce, 40000)
        assert e.value.code == abi.CODE["INVALID_NORMALIZATION"]
    else:
        got, _ = routability.register_clustering_areas(xy, cl, ce, 40000)
        assert np.all(np.isfinite(got)) and got[0] == pytest.approx(expected[0], rel=1e-12)
