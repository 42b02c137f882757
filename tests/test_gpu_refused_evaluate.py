"""An evaluation that is refused for a coordinate that is not finite leaves the
handle as it was: the run that goes on afterwards gives the coordinates, targets
and counters of a run without it, on both engines."""
from contextlib import nullcontext

import numpy as np
import pytest

from test_gpu_no_spare_memory import FullPool
from texo_gb300 import abi, problem as P
from texo_gb300.placer import Placer, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [abi.ENGINE_HOST, abi.ENGINE_DEVICE])
@pytest.mark.parametrize("first", [0, 1, 5])
def test_a_refused_evaluation_leaves_the_run_as_it_was(engine, first):
    prob = P.synthetic(48, 2000, 60, 2400, 6.0, 3)
    prm = default_params(engine=engine, best_effort=1, max_iterations=40)

    def run(refused):
        with Placer(prob, prm) as g:
            if first:
                g.run(first, allow_nonconverged=True)
            for k in refused:
                c, _, _ = g.initial()
                c[k] = np.nan
                with pytest.raises(abi.TexoGpError) as e:
                    g.evaluate(c, 4.0)
                assert e.value.code == abi.CODE["NONFINITE_UNIT_COORDINATE"]
            t, x, s = g.run(4, allow_nonconverged=True)
        s.pop("elapsed_ms")
        return t, x, s

    plain, after = run([]), run([0, 2000, -1])
    assert np.array_equal(plain[0], after[0]) and np.array_equal(plain[1], after[1])
    assert plain[2] == after[2]


@pytest.mark.parametrize("engine", [abi.ENGINE_HOST, abi.ENGINE_DEVICE])
@pytest.mark.parametrize("first", [0, 2])
@pytest.mark.parametrize("spare", [True, False])
def test_more_coordinates_than_the_host_checks(engine, first, spare):
    """Beyond 1 MiB of coordinates the device flags them, or the host where there is no memory to stage them."""
    prob = P.synthetic(290, 70000, 300, 80000, 6.0, 1)
    prm = default_params(engine=engine, best_effort=1, max_iterations=40, bins_x=256, bins_y=256)

    def run(refused):
        with Placer(prob, prm) as g:
            c, _, _ = g.initial()
            assert c.size > 1 << 17
            if first:
                g.run(first, allow_nonconverged=True)
            with nullcontext() if spare else FullPool():
                for k, value in refused:
                    bad = c.copy()
                    bad[k] = value
                    with pytest.raises(abi.TexoGpError) as e:
                        g.evaluate(bad, 4.0, arrays=False)
                    assert e.value.code == abi.CODE["NONFINITE_UNIT_COORDINATE"]
            t, x, s = g.run(3, allow_nonconverged=True)
            wirelength = g.evaluate(x, 4.0, arrays=False)["wirelength"]
        s.pop("elapsed_ms")
        return t, x, s, wirelength

    plain, after = run([]), run([(0, np.nan), (70000, np.inf), (-1, -np.inf)])
    assert np.array_equal(plain[0], after[0]) and np.array_equal(plain[1], after[1])
    assert plain[2:] == after[2:]
