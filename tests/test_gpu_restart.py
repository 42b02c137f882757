"""Steps that restart behind an extrapolated point that differs from the
origin: the host engine, which has evaluated that point ahead, then goes back to
the origin's residual and gradient. Both engines, whose controllers are written
apart, give the same coordinates, targets and counts, bit for bit; the trace
shows that steps did restart (their momentum begins again at the golden ratio)."""
import numpy as np
import pytest

from texo_gb300 import abi, problem as P
from texo_gb300.placer import Placer, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,ulps,expected", [(0, 0.0, 3), (0, 1.0, 1), (1, 64.0, 1), (2, 0.0, 4)])
def test_restarted_steps_are_the_same_on_both_engines(seed, ulps, expected):
    prob = P.synthetic(24, 60, 12, 80, 6.0, seed)
    runs, restarts = [], 0
    for engine in (abi.ENGINE_HOST, abi.ENGINE_DEVICE):
        prm = default_params(engine=engine, best_effort=1, max_iterations=200, overflow_target_override=1e-4,
                             initial_density_weight=1e-6, alpha_low=1.00001, alpha_high=1.00002,
                             objective_margin_ulps=ulps)
        with Placer(prob, prm) as g:
            runs.append(g.run(200, allow_nonconverged=True))
            if engine == abi.ENGINE_HOST:
                golden = (1 + np.sqrt(5.0)) / 2
                restarts = sum(r.iteration > 1 and abs(r.momentum - golden) < 1e-12 for r in g.trace())
    (ta, xa, sa), (tb, xb, sb) = runs
    assert restarts == expected
    assert np.array_equal(ta, tb) and np.array_equal(xa, xb)
    for k in ("iterations", "evaluations", "density_evaluations", "line_search_trials"):
        assert sa[k] == sb[k], k
