"""Lattices cut into runs of 256 consecutive subvolumes instead of bricks (geo_rows): both sides of each line of the
rule, last runs that are full, one short of full and a single subvolume; small and network models, resident and phase
kernels, slabs and learned classification on such lattices, batches of uneven replicas.  Bit for bit."""
import numpy as np
import pytest

from helpers import assert_same, bits

pytestmark = pytest.mark.gpu


def _schlogl(dims, seed=3):
    from pliscuda_b200 import workloads
    m = workloads._model(dims, 1, [({0: 2}, {0: 3}), ({0: 3}, {0: 2}), ({}, {0: 1}), ({0: 1}, {})],
                         [0.03, 1e-4, 200.0, 3.5], [1.0])
    n = dims[0] * dims[1] * dims[2]
    st = np.random.default_rng(seed).poisson(120, n)
    st[::97] = 4  # critical subvolumes
    return m, st.astype(np.uint32)


def _network(dims, seed=3):
    from pliscuda_b200 import workloads
    s = 6
    rx = [({}, {0: 1})] + [({i: 1}, {i + 1: 1}) for i in range(s - 1)] + [({s - 1: 1}, {})]
    m = workloads._model(dims, s, rx, [40.0] + [1.0] * s, [0.5] * s)
    return m, np.random.default_rng(seed).poisson(40, s * dims[0] * dims[1] * dims[2]).astype(np.uint32)


# x*y*z: 4096 is the least number of subvolumes that runs take
@pytest.mark.parametrize("dims,steps", [
    ((17, 15, 16), 5),    # 4080: bricks
    ((17, 241, 1), 5),    # 4097: 17 runs, the last of one subvolume
    ((13, 21, 15), 5),    # 4095: bricks, one below
    ((1, 4111, 1), 5),    # one subvolume wide
    ((43, 41, 42), 2),    # resident as runs, not as bricks; phase kernels below three steps
    ((43, 41, 42), 4),
    ((128, 64, 10), 3),   # runs of parts of x rows, phase kernels
    ((256, 300, 1), 3),   # a run is an x row
    ((16, 16, 297), 3),   # a run is a layer
    ((51, 45, 35), 3),    # phase kernels, 80325 = 313 runs and 197
])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_small_model(dims, steps, precision):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    m, st = _schlogl(dims)
    with Simulation(m, seed=7, precision=precision) as sim, Simulation(m, seed=7, precision=precision, tile=(8, 8, 4)) as old:
        for s in (sim, old):
            s.set_state(st)
            s.step(steps)
        assert_same(sim, old, f"{dims} runs and bricks")
        if precision == "fp64":
            orc = Oracle.from_model(m, seed=7)
            orc.set_state(st)
            orc.step(steps)
            assert_same(sim, orc, f"{dims}")


@pytest.mark.parametrize("dims", [(17, 241, 1), (50, 61, 29), (43, 41, 42)])
def test_network(dims):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    m, st = _network(dims)
    with Simulation(m, seed=7) as sim:
        orc = Oracle.from_model(m, seed=7)
        for s in (sim, orc):
            s.set_state(st)
            s.step(3)
        assert_same(sim, orc, f"{dims}")


def test_slabs_are_bricks():
    from test_slabs_gpu import _compare
    m, st = _schlogl((19, 21, 18))
    assert _compare(m, st, [(0, 8), (8, 18)], 0.02, seed=5).steps > 3


def test_learned_on_and_off():
    """A proposer attached, detached and attached again: the same sequence on a lattice of runs and on bricks."""
    from pliscuda_b200 import Simulation
    from test_learned_gpu import random_weights
    m, st = _schlogl((43, 41, 42))
    with Simulation(m, mode="corrected", seed=7) as sim, Simulation(m, mode="corrected", seed=7, tile=(8, 8, 4)) as old:
        for s in (sim, old):
            s.set_state(st)
        for on in (True, False, True, False):
            for s in (sim, old):
                s.set_proposer(random_weights(2) if on else None, 8.0)
                s.step(4)
            assert_same(sim, old, f"proposer {on}")


@pytest.mark.parametrize("learned", [False, True])
def test_uneven_batch(learned):
    from pliscuda_b200 import Simulation
    from pliscuda_b200.batch import Batch
    from test_learned_gpu import random_weights
    dims = [(1, 1, 1), (8, 8, 4), (16, 16, 1), (257, 1, 1), (9, 9, 5), (5, 51, 1), (17, 16, 16), (3, 2, 7)]
    models = [_schlogl(d, seed=i) for i, d in enumerate(dims)]
    w = random_weights(2)
    b = Batch.from_models([m for m, _ in models], mode="corrected", seed=11)
    if learned:
        b.set_proposer(w, 8.0)
    for r, (_, st) in enumerate(models):
        b.set_state(r, st)
    b.step(12)
    for r, (m, st) in enumerate(models):
        with Simulation(m, mode="corrected", seed=11, replica=r, tile=(8, 8, 4), learned_mlp="mma.sync") as s:
            if learned:
                s.set_proposer(w, 8.0)
            s.set_state(st)
            s.step(12)
            assert np.array_equal(b.get_state(r), s.get_state()), f"replica {r}"
            x, y = b.stats(r), s.stats()
            assert bits(np.array([x.time]))[0] == bits(np.array([y.time]))[0]
            assert (x.steps, x.events, x.rollbacks) == (y.steps, y.events, y.rollbacks)
    b.close()
