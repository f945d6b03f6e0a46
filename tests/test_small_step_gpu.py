"""The small-model kernels (pliscuda_b200/csrc/small_step.cuh) against the oracle, bit for bit, where
they can go wrong: lattices with sides of 1, 2 and 3 (subvolumes with 0 to 6 neighbours, neighbours with
fewer than six of their own), bricks that do not fill, one to four species, every reaction order,
means on both sides of the inversion limit, counts around the critical threshold, neighbour tables, and
enough draws for the uniforms next to 1 that the binary32 search treats apart."""
import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

NETS = {
    # reactions, rates, jump rates, mean counts
    "schlogl": ([({0: 2}, {0: 3}), ({0: 3}, {0: 2}), ({}, {0: 1}), ({0: 1}, {})], [0.03, 1e-4, 200.0, 3.5], [1.0], [300]),
    "scarce": ([({0: 1}, {1: 1}), ({1: 2}, {0: 1}), ({}, {0: 1}), ({0: 1, 1: 1}, {})], [0.4, 0.05, 3.0, 0.02],
               [0.3, 0.0], [9, 14]),
    "brusselator": ([({}, {0: 1}), ({0: 1}, {1: 1}), ({0: 2, 1: 1}, {0: 3}), ({0: 1}, {})], [100.0, 300.0, 1e-4, 1.0],
                    [0.5, 2.0], [100, 30000]),
    "three": ([({0: 1, 1: 1}, {2: 1}), ({2: 1}, {0: 1, 1: 1}), ({2: 3}, {0: 1})], [0.01, 0.5, 1e-4], [0.1, 0.2, 0.0],
              [40, 60, 25]),
    "four": ([({0: 1, 1: 1, 2: 1}, {3: 2}), ({3: 2}, {0: 1}), ({1: 1}, {2: 1}), ({}, {1: 4, 2: 1})],
             [1e-3, 0.02, 0.3, 5.0], [0.1, 0.7, 0.2, 1.5], [30, 50, 20, 60]),
    "fast_jumps": ([({}, {0: 1}), ({0: 1}, {})], [1.0, 1e-3], [50.0], [4000]),
}
LATTICES = [(1, 1, 1), (7, 1, 1), (2, 1, 3), (3, 2, 2), (5, 4, 3), (9, 9, 5), (17, 3, 10)]


def _model(name, dims, seed):
    from pliscuda_b200 import workloads
    reactions, rates, jumps, means = NETS[name]
    m = workloads._model(dims, len(jumps), reactions, rates, jumps)
    rng = np.random.default_rng(seed)
    st = np.concatenate([rng.poisson(v, m.n_subvolumes) for v in means]).astype(np.uint32)
    return m, st


def _pair(m, st, mode, precision, **kw):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    sim = Simulation(m, mode=mode, precision=precision, seed=77, **kw)
    orc = Oracle.from_model(m, seed=77, mode=mode, precision=precision, **{k: v for k, v in kw.items() if k == "critical_threshold"})
    sim.set_state(st)
    orc.set_state(st)
    return sim, orc


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", sorted(NETS))
def test_small_models_on_awkward_lattices(name, mode, precision):
    for dims in LATTICES:
        m, st = _model(name, dims, sum(dims))
        sim, orc = _pair(m, st, mode, precision)
        assert_same(sim, orc, f"{dims} start")
        for n in (1, 1, 6):
            sim.step(n)
            orc.step(n)
            assert_same(sim, orc, f"{dims} after {n} more steps")
        sim.close()


@pytest.mark.parametrize("threshold", [0, 1, 10, 1000])
@pytest.mark.parametrize("mode", [0, 1])
def test_critical_thresholds(mode, threshold):
    m, st = _model("scarce", (6, 5, 4), 3)
    sim, orc = _pair(m, st, mode, 0, critical_threshold=threshold)
    for _ in range(5):
        sim.step(1)
        orc.step(1)
        assert_same(sim, orc, f"threshold {threshold}")
    sim.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_binary32_uniforms_next_to_one(mode):
    """1.3 M subvolume-draws: about 40 uniforms above 1 - 2^-15, where the search keeps its tail test."""
    m, st = _model("schlogl", (32, 32, 16), 5)
    sim, orc = _pair(m, st, mode, 1)
    for _ in range(8):
        sim.step(1)
        orc.step(1)
        assert_same(sim, orc)
    sim.close()


@pytest.mark.parametrize("jump", [0.0, 1e-300, 1e-40, 1e30])
def test_extreme_jump_rates(jump):
    """Rates too small or too large for the neighbour division of the small-model kernels take the generic ones."""
    from pliscuda_b200 import workloads
    m = workloads._model((5, 4, 3), 1, [({}, {0: 1}), ({0: 1}, {})], [5.0, 0.1], [jump])
    st = np.random.default_rng(1).poisson(50, m.n_subvolumes).astype(np.uint32)
    sim, orc = _pair(m, st, 0, 0)
    for _ in range(3):
        sim.step(1)
        orc.step(1)
        assert_same(sim, orc, f"jump rate {jump}")
    sim.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_neighbour_table(mode, precision):
    """A ring with chords as a table: 2 to 6 neighbours in file order, not a lattice."""
    from pliscuda_b200 import Model
    n, rng = 300, np.random.default_rng(2)
    adj = [{(c - 1) % n, (c + 1) % n} for c in range(n)]
    for _ in range(400):
        a, b = (int(v) for v in rng.integers(n, size=2))
        if a != b and b not in adj[a] and len(adj[a]) < 6 and len(adj[b]) < 6:
            adj[a].add(b)
            adj[b].add(a)
    nb = np.array([sorted(v) + [c] * (6 - len(v)) for c, v in enumerate(adj)], np.uint32)
    reactions, rates, jumps, means = NETS["scarce"]
    base, _ = _model("scarce", (2, 2, 2), 0)
    m = Model(n_subvolumes=n, n_species=2, n_reactions=4, reactants=base.reactants, products=base.products,
              reaction_rates=rates, diffusion_rates=jumps, neighbours=nb.reshape(-1))
    st = np.concatenate([rng.poisson(v, n) for v in means]).astype(np.uint32)
    sim, orc = _pair(m, st, mode, precision)
    for _ in range(8):
        sim.step(1)
        orc.step(1)
        assert_same(sim, orc)
    sim.close()
