"""Rate constants beyond the range of binary32 in the FP32 form: inf for the device, so that a reaction whose
reactant is missing has the propensity inf x 0 = NaN.  Corrected semantics leave out every propensity that is not
positive; the step follows the binary32 oracle bit for bit, for a handle of a small model, one of a network and a
batch in which one replica has such a rate."""
import numpy as np
import pytest

from helpers import assert_same, bits

pytestmark = pytest.mark.gpu


def _model(S, top, dims=(5, 4, 3)):
    from pliscuda_b200 import workloads
    rx = [({}, {0: 1}), ({0: 1}, {}), ({1: 2}, {})] + [({i: 1}, {}) for i in range(2, S)]
    m = workloads._model(dims, S, rx, [50.0, 1.0, top] + [1.0] * (S - 2), [0.3] * S)
    n = m.n_subvolumes
    st = np.random.default_rng(4).poisson(50, S * n).astype(np.uint32).reshape(S, n)
    st[1] = 0  # the third reaction never has its reactant
    return m, st.reshape(-1)


# 3.4028235677973366e38 is the least binary64 value that rounds to inf in binary32
@pytest.mark.parametrize("top", [1e39, 3.4028235677973366e38, 3.4028235e38])
@pytest.mark.parametrize("S", [2, 6], ids=["small", "network"])
def test_rates_beyond_binary32(S, top):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    m, st = _model(S, top)
    with Simulation(m, seed=7, mode=1, precision=1) as sim:
        orc = Oracle.from_model(m, seed=7, mode=1, precision=1)
        for s in (sim, orc):
            s.set_state(st)
        assert_same(sim, orc, "start")
        for n in (1, 4):
            sim.step(n)
            orc.step(n)
            assert_same(sim, orc, f"after {n} more steps")


def test_one_replica_of_a_batch():
    from oracle.oracle import Oracle
    from pliscuda_b200.batch import Batch
    models = [_model(2, 1.0), _model(2, 1e39)]
    with Batch.from_models([m for m, _ in models], seed=7, mode=1, precision=1) as b:
        for r, (_, st) in enumerate(models):
            b.set_state(r, st)
        b.step(5)
        for r, (m, st) in enumerate(models):
            orc = Oracle.from_model(m, seed=7, mode=1, precision=1, replica=r)
            orc.set_state(st)
            orc.step(5)
            assert np.array_equal(b.get_state(r), orc.get_state()), f"replica {r}"
            assert bits(np.array([b.stats(r).time]))[0] == bits(np.array([orc.stats().time]))[0]
