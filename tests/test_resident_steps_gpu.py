"""The persistent step kernel of small systems (k_steps in pliscuda_b200/csrc/engine_kernels.cuh) against the
phase kernels (a handle with its own wait limit keeps them) and the oracle: one CTA to as many as the GPU
holds, one more, runs that end within a launch and after several, steps mixed with runs, rollbacks, critical
and exact events, and a state continued from one to the other.  Bit for bit."""
import numpy as np
import pytest

from helpers import assert_same, bits, random_graph_model
from test_net_step_gpu import _network
from test_small_step_gpu import _model

pytestmark = pytest.mark.gpu


def _both(m, st, mode, precision, plan, **kw):
    from pliscuda_b200 import Simulation
    out = []
    for polls in (0, 1 << 30):
        with Simulation(m, mode=mode, precision=precision, seed=8, wait_polls=polls, **kw) as sim:
            sim.set_state(st)
            seen = []
            for what, v in plan:
                s = sim.run(v) if what == "run" else sim.step(v)
                tau, fl = sim.taus()
                seen.append((sim.get_state(), bits(tau), fl, bits(np.array([s.time])), s.steps, s.rollbacks, s.events,
                             s.exact_events, s.stop_reason))
            out.append(seen)
    for k, (a, b) in enumerate(zip(*out)):
        for x, y in zip(a, b):
            assert np.array_equal(x, y), (k, plan[k])


PLAN = [("step", 6), ("step", 1), ("step", 37), ("step", 5), ("step", 20)]


@pytest.mark.parametrize("dims", [(1, 1, 1), (8, 8, 4), (9, 8, 4), (20, 19, 7), (33, 21, 10), (40, 40, 40), (48, 48, 32), (48, 48, 36)])
@pytest.mark.parametrize("mode", [0, 1])
def test_small_models_of_growing_size(dims, mode):
    m, st = _model("schlogl", dims, 1)
    _both(m, st, mode, 0, PLAN)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_events_of_every_kind(mode, precision):
    m, st = _model("scarce", (13, 9, 5), 2)
    _both(m, st, mode, precision, PLAN + [("step", 300)])
    m, st = _network(6, 12, 4, (12, 11, 6), 2)
    _both(m, st, mode, precision, PLAN)
    m, st = random_graph_model(700, 5)
    _both(m, st, mode, precision, PLAN)


@pytest.mark.parametrize("mode", [0, 1])
def test_runs_to_a_time(mode):
    from pliscuda_b200 import Simulation
    m, st = _model("schlogl", (10, 7, 6), 3)
    with Simulation(m, mode=mode, seed=8) as sim:
        sim.set_state(st)
        t = sim.step(100).time
    _both(m, st, mode, 0, [("run", 0.3 * t), ("run", 0.3 * t), ("step", 6), ("run", t), ("run", 0.0)])


def test_more_attempts_than_a_launch_takes():
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    m, st = _model("scarce", (3, 3, 2), 4)
    with Simulation(m, seed=8) as sim:
        sim.set_state(st)
        sim.step(9001)
        orc = Oracle.from_model(m, seed=8)
        orc.set_state(st)
        orc.step(9001)
        assert_same(sim, orc)


@pytest.mark.parametrize("mode", [0, 1])
def test_rollbacks(mode):
    """Means far above the counts that feed them: attempts with negative counts are discarded."""
    from pliscuda_b200 import workloads
    m = workloads._model((6, 5, 4), 2, [({0: 1}, {1: 1}), ({1: 2}, {}), ({}, {0: 3})], [40.0, 3.0, 60.0], [30.0, 0.1])
    st = np.random.default_rng(6).poisson(14, 2 * m.n_subvolumes).astype(np.uint32)
    _both(m, st, mode, 0, PLAN, epsilon=0.9, critical_threshold=2, max_rollbacks=200)
    _both(m, st, mode, 0, PLAN, epsilon=0.9, critical_threshold=2, max_rollbacks=200, pooled_draws=1)
