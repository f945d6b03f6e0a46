"""Batches of steps without the exact-event kernels (Engine::advance) against the oracle on lattices too large for
the persistent kernel: systems in which exact events never come, come in every step, and come and go, so that
batches stop and are resumed with the kernels; both semantics, single steps in between.  Bit for bit."""
import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

DIMS = (48, 48, 36)  # 324 bricks of 256: more than two per SM


def _case(name):
    from pliscuda_b200 import workloads
    rng = np.random.default_rng(3)
    n = DIMS[0] * DIMS[1] * DIMS[2]
    if name == "none":
        m = workloads._model(DIMS, 1, [({}, {0: 1}), ({0: 1}, {})], [50.0, 1.0], [0.5])
        return m, rng.poisson(50, n).astype(np.uint32)
    if name == "always":
        m = workloads._model(DIMS, 2, [({0: 1}, {1: 1}), ({1: 1}, {0: 1})], [0.4, 0.2], [0.3, 0.1])
        return m, rng.poisson(9, 2 * n).astype(np.uint32)
    # a decaying species in one corner passes the critical threshold now and then
    m = workloads._model(DIMS, 2, [({}, {0: 1}), ({0: 1}, {}), ({1: 1}, {})], [80.0, 1.0, 0.3], [0.5, 0.0])
    st = np.concatenate([rng.poisson(80, n), np.zeros(n)]).astype(np.uint32)
    st[n:n + 3] = (14, 22, 60)
    return m, st


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", ["none", "always", "sometimes"])
def test_batches_with_and_without_exact_events(name, mode):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    m, st = _case(name)
    with Simulation(m, mode=mode, seed=12) as sim:
        orc = Oracle.from_model(m, seed=12, mode=mode)
        sim.set_state(st)
        orc.set_state(st)
        for n in (40, 3, 70, 33):
            sim.step(n)
            orc.step(n)
            assert_same(sim, orc, f"{name} after {n} more steps")
        t = sim.stats().time
        sim.run(1.5 * t)
        orc.run(1.5 * t)
        assert_same(sim, orc, f"{name} run")
        events = sim.stats().exact_events
        assert (events == 0) == (name == "none")
