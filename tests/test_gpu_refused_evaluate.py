"""An evaluation that is refused for a coordinate that is not finite leaves the
handle as it was: the run that goes on afterwards gives the coordinates, targets
and counters of a run without it, on both engines."""
import numpy as np
import pytest

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
