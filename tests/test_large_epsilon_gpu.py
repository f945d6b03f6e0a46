"""Tolerances far above 1 in a network's classification, which ranks the species' leap bounds in binary32 before it
computes the smallest in full: a species whose drift cancels, so that its bound is the spread's, (epsilon x)^2 / s2,
beside one with a drift bound above it.  Both sides of the largest epsilon whose square stays within binary32 for
every count (1e9), against the oracle bit for bit."""
import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("epsilon", [0.05, 1.0, 1e9, 1.0000001e9, 1e12, 1e30])
def test_spread_bound_below_a_drift_bound(epsilon, mode, precision):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation, workloads
    x0, x1 = 500000000, 100000000
    # species 0: 1e13 - 2e4 x0 + 1e-8, drift 1e-8 and spread 2e13; species 1: drift bound 2.4 times its spread bound
    spread0 = (epsilon * x0) ** 2 / 2e13
    m = workloads._model((2, 1, 1), 5, [({}, {0: 1}), ({0: 1}, {}), ({}, {0: 1}), ({1: 1}, {})],
                         [1e13, 2e4, 1e-8, epsilon / (2.4 * spread0)], [0.0] * 5)
    st = np.zeros((5, 2), np.uint32)
    st[0], st[1] = x0, x1
    with Simulation(m, seed=7, mode=mode, precision=precision, epsilon=epsilon) as sim:
        orc = Oracle.from_model(m, seed=7, mode=mode, precision=precision, epsilon=epsilon)
        for s in (sim, orc):
            s.set_state(st.reshape(-1))
        assert_same(sim, orc, f"epsilon {epsilon}")
