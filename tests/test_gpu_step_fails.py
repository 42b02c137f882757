"""A step of the host engine that fails behind an extrapolated point (here for
filler charges beyond FP32, whose preconditioner is refused) leaves a run that
can go on: with the charges put back the next steps are those of a run
without the failure, bit for bit."""
import numpy as np
import pytest

from texo_gb300 import abi, problem as P
from texo_gb300.placer import Placer, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [1, 2, 6])
def test_a_run_goes_on_after_a_failed_step(first):
    prob = P.synthetic(48, 2000, 60, 2400, 6.0, 3)

    def run(fails):
        with Placer(prob, default_params(engine=abi.ENGINE_HOST, best_effort=1, max_iterations=60)) as g:
            _, charge = g.fillers()
            assert charge.size > 0
            g.run(first, allow_nonconverged=True)
            if fails:
                g.set_charges(filler_charge=np.full(charge.size, 1e300))
                with pytest.raises(abi.TexoGpError) as e:
                    g.run(1, allow_nonconverged=True)
                assert e.value.code == abi.CODE["INVALID_NORMALIZATION"]
            g.set_charges(filler_charge=charge)
            return g.run(4, allow_nonconverged=True)

    plain, after = run(False), run(True)
    assert np.array_equal(plain[0], after[0]) and np.array_equal(plain[1], after[1])
    assert plain[2]["objective"] == after[2]["objective"]
