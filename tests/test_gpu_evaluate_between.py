"""An evaluation of other coordinates between two parts of a run, and one that is
refused, leave the run as it is, on both engines: the steps behind it, the first
of which restarts and goes back to the origin's kept field gradients, give the
coordinates and targets of the run without it, bit for bit; after a refused one
the counts are the same too."""
import numpy as np
import pytest

from texo_gb300 import abi, problem as P
from texo_gb300.placer import Placer, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [abi.ENGINE_HOST, abi.ENGINE_DEVICE])
@pytest.mark.parametrize("seed,ulps,restart", [(0, 1.0, 100), (1, 64.0, 68), (2, 1.0, 65)])
def test_a_run_goes_on_behind_an_evaluation(engine, seed, ulps, restart):
    prob = P.synthetic(24, 60, 12, 80, 6.0, seed)
    prm = default_params(engine=engine, best_effort=1, max_iterations=200, overflow_target_override=1e-4,
                         initial_density_weight=1e-6, alpha_low=1.00001, alpha_high=1.00002,
                         objective_margin_ulps=ulps)

    def run(between):
        with Placer(prob, prm) as g:
            g.run(restart - 1, allow_nonconverged=True)
            c, _, _ = g.initial()
            if between == "evaluated":
                g.evaluate(c[::-1].copy(), 3.0)
            elif between == "refused":
                c[5] = np.nan
                with pytest.raises(abi.TexoGpError):
                    g.evaluate(c[::-1].copy(), 3.0)
            t, x, s = g.run(8, allow_nonconverged=True)
            if engine == abi.ENGINE_HOST:
                golden = (1 + np.sqrt(5.0)) / 2
                assert abs(g.trace()[restart - 1].momentum - golden) < 1e-12
        return t, x, [s[k] for k in ("iterations", "evaluations", "density_evaluations", "line_search_trials")]

    plain, evaluated, refused = run(None), run("evaluated"), run("refused")
    for other in (evaluated, refused):
        assert np.array_equal(plain[0], other[0]) and np.array_equal(plain[1], other[1])
    assert plain[2] == refused[2]
