"""Neighbour tables with one-way edges into a subvolume that has no neighbours of its own.  The reference divides a
neighbour's jumps by that neighbour's count of neighbours (tau.cu:120-136), here 0: the quotient is NaN while the sink
is empty and inf after that, and the step follows the oracle bit for bit with either, for a model that fits the small
tables and one that fits the network tables, with and without compartments."""
import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


def _chain_into_sink(n, S, R, compartments, in_sink):
    from pliscuda_b200 import Model
    nb = np.zeros(6 * n, np.uint32)
    for c in range(n):  # the last subvolume is the sink, the first one a source without a way back
        row = [] if c == n - 1 else [c + 1] + ([c - 1] if c > 1 else [])
        nb[6 * c:6 * c + 6] = row + [c] * (6 - len(row))
    re, pr = np.zeros((S, R), np.int32), np.zeros((S, R), np.int32)
    for i in range(min(S, R)):
        re[i, i] = 1
    C = 2 if compartments else 1
    m = Model(n_subvolumes=n, n_species=S, n_reactions=R, reactants=re.reshape(-1), products=pr.reshape(-1),
              reaction_rates=[0.1, 0.2][:C] * R, diffusion_rates=[0.3] * (C * S), neighbours=nb, n_compartments=C,
              compartment=np.arange(n, dtype=np.int32) % 2 if compartments else None)
    st = np.random.default_rng(5).poisson(60, S * n).astype(np.uint32).reshape(S, n)
    st[:, n - 1] = in_sink
    return m, st.reshape(-1)


@pytest.mark.parametrize("in_sink", [0, 20])
@pytest.mark.parametrize("compartments", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("S,R", [(1, 1), (6, 6)], ids=["small", "network"])
def test_one_way_edges_into_a_sink(S, R, mode, precision, compartments, in_sink):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    m, st = _chain_into_sink(40, S, R, compartments, in_sink)
    with Simulation(m, seed=7, mode=mode, precision=precision) as sim:
        orc = Oracle.from_model(m, seed=7, mode=mode, precision=precision)
        for s in (sim, orc):
            s.set_state(st)
        assert_same(sim, orc, "start")
        for n in (1, 3, 5):
            sim.step(n)
            orc.step(n)
            assert_same(sim, orc, f"after {n} more steps")
