"""The tcgen05 MLP's waits with a short limit (plis_options.wait_polls): a group of threads whose wait runs out
stops as a whole, after the same layer, so the classification ends and the call reports PLIS_ERR_TIMEOUT; where
no wait runs out the results are those of the default limit, bit for bit.  Either way the handle still answers
and the next one, with the default limit, runs as before."""
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


# fewer tiles of 128 subvolumes than a CTA has groups, a few CTAs, several tiles per group
@pytest.mark.parametrize("side", [5, 16, 60])
@pytest.mark.parametrize("polls", [1, 2, 3])
def test_short_limits_end(side, polls):
    from pliscuda_b200 import PlisError, Simulation, workloads
    from test_learned_gpu import random_weights
    m, st = workloads.schlogl(side)

    def learned(**kw):
        sim = Simulation(m, mode="corrected", seed=5, **kw)
        sim.set_proposer(random_weights(1), 8.0)
        sim.set_state(st)
        return sim

    with learned() as ref, learned(wait_polls=polls) as short:
        ref.step(6)
        try:
            short.step(6)
            assert_same(short, ref, f"{side}^3")
        except PlisError as e:
            assert e.status == 6, e  # PLIS_ERR_TIMEOUT
            assert short.stats().status == 6
    with learned() as again, learned() as ref:
        again.step(6)
        ref.step(6)
        assert_same(again, ref, f"{side}^3 afterwards")
