"""The network kernels (pliscuda_b200/csrc/net_step.cuh) against the oracle, bit for bit, at the edges of
their range: 1 to 16 species and 5 to 32 reactions of order 0 to 3, pooled and per-channel draws,
several compartments on lattices and neighbour tables, lattices with sides of 1 to 3, draws above the
32-bit net changes, networks just beyond the tables (generic kernels), and the event log."""
import numpy as np
import pytest

from helpers import assert_same, birth_death_model, random_graph_model

pytestmark = pytest.mark.gpu

LATTICES = [(1, 1, 1), (5, 1, 2), (3, 3, 2), (9, 5, 6)]


def _network(S, R, seed, dims, compartments=1, mean=25):
    from pliscuda_b200 import Model
    rng = np.random.default_rng(seed)
    n = dims[0] * dims[1] * dims[2]
    re = np.zeros((S, R), np.int32)
    pr = np.zeros((S, R), np.int32)
    rates = np.zeros((compartments, R))
    for r in range(R):
        order = int(rng.integers(0, 4))
        for s in rng.integers(S, size=order):
            re[s, r] += 1
        for s in rng.integers(S, size=int(rng.integers(0, 3))):
            pr[s, r] += 1
        if (re[:, r] == pr[:, r]).all():
            pr[0, r] += 1
        rates[:, r] = 10 ** rng.uniform(-1, 1, compartments) / float(mean) ** max(0, order - 1)
    m = Model(n_subvolumes=n, n_species=S, n_reactions=R, reactants=re.reshape(-1), products=pr.reshape(-1),
              reaction_rates=rates.reshape(-1), diffusion_rates=rng.uniform(0, 1, compartments * S), lattice=dims,
              n_compartments=compartments,
              compartment=rng.integers(compartments, size=n).astype(np.int32) if compartments > 1 else None)
    st = rng.poisson(rng.uniform(2, 2 * mean, S)[:, None], (S, n)).astype(np.uint32).reshape(-1)
    return m, st


def _pair(m, st, mode, precision, **kw):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    sim = Simulation(m, mode=mode, precision=precision, seed=41, **kw)
    orc = Oracle.from_model(m, seed=41, mode=mode, precision=precision, **kw)
    sim.set_state(st)
    orc.set_state(st)
    return sim, orc


def _compare(sim, orc, steps, where=""):
    assert_same(sim, orc, f"{where} start")
    for n in steps:
        sim.step(n)
        orc.step(n)
        assert_same(sim, orc, f"{where} after {n} more steps")
    sim.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("S,R", [(1, 5), (2, 9), (5, 12), (16, 32), (17, 12), (6, 33)])
def test_networks_on_awkward_lattices(S, R, mode, precision):
    for dims in LATTICES:
        m, st = _network(S, R, 100 * S + R, dims)
        _compare(*_pair(m, st, mode, precision), (1, 1, 4), str(dims))


@pytest.mark.parametrize("pooled", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("S,R", [(2, 3), (5, 12)])
def test_pooled_and_per_channel_draws(S, R, mode, pooled):
    m, st = _network(S, R, 7, (6, 7, 3))
    _compare(*_pair(m, st, mode, 0, pooled_draws=pooled), (1, 6))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_pool_events(mode, precision):
    m, st = birth_death_model(side=9)
    _compare(*_pair(m, st, mode, precision), (1, 7))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("compartments", [2, 32, 33])
def test_compartments(compartments, mode, precision):
    m, st = _network(4, 4, 5, (7, 5, 4), compartments)
    _compare(*_pair(m, st, mode, precision), (1, 6), "lattice")


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_neighbour_table(mode, precision):
    m, st = random_graph_model(300, 3)
    _compare(*_pair(m, st, mode, precision), (1, 7))


@pytest.mark.parametrize("start", [700_000_000, (1 << 30) - 1_000_000])
@pytest.mark.parametrize("rate", [1e10, 1e12])
def test_net_changes_beyond_32_bits(rate, start):
    """Immigration far above the jumps: from a count of 7e8 a leap draws 3e7 (above 2^24), from just below
    2^30 the guards roll the attempts back."""
    from oracle.oracle import Oracle
    from pliscuda_b200 import PlisError, Simulation, workloads
    m = workloads._model((3, 2, 2), 5, [({}, {i: 1}) for i in range(5)] + [({i: 1}, {}) for i in range(5)],
                         [rate] * 5 + [0.5] * 5, [1.0] * 5)
    st = np.full(5 * 12, start, np.uint32)
    sim = Simulation(m, seed=3, max_rollbacks=6)
    orc = Oracle.from_model(m, seed=3, max_rollbacks=6)
    sim.set_state(st)
    orc.set_state(st)
    for _ in range(3):
        status = 0
        try:
            sim.step(1)
        except PlisError as e:
            status = e.status
        assert status == orc.step(1)  # the oracle returns its status
        if status:
            assert status == 7 and start > 1 << 29  # PLIS_ERR_STUCK
            break
        assert_same(sim, orc, f"rate {rate}")
    sim.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_event_log(mode):
    m, st = _network(5, 12, 9, (6, 5, 4))
    sim, orc = _pair(m, st, mode, 0)
    sim.set_event_log(1 << 16)
    before = sim.stats().events
    sim.step(5)
    orc.step(5)
    rec, dropped = sim.read_event_log()
    assert dropped == 0
    exact = rec["kind"] >= 3
    assert int(rec["count"].astype(np.int64).sum()) == sim.stats().events - before
    assert int(exact.sum()) == sim.stats().exact_events
    assert_same(sim, orc)
    sim.close()
