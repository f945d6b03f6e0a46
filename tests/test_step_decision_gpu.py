"""The step decision's kernel (k_control) around its 512 threads: one classification record, a CTA's worth less one,
exactly, one more, and three per thread less one; the subvolume that sets the step lies in the last record.  Small
and network models against the oracle, bit for bit."""
import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


def _model(kind, dims):
    from pliscuda_b200 import workloads
    if kind == "small":
        return workloads._model(dims, 1, [({}, {0: 1}), ({0: 1}, {})], [4000.0, 1.0], [0.05])
    s = 6  # a chain of more species than the small-model kernels take
    rx = [({}, {0: 1})] + [({i: 1}, {i + 1: 1}) for i in range(s - 1)] + [({s - 1: 1}, {})]
    return workloads._model(dims, s, rx, [4000.0] + [1.0] * s, [0.05] * s)


@pytest.mark.parametrize("records", [1, 511, 512, 513, 1535])
@pytest.mark.parametrize("kind", ["small", "net"])
def test_decision_over_records(kind, records):
    from oracle.oracle import Oracle
    from pliscuda_b200 import Simulation
    m = _model(kind, (8, 8, 4 * records))  # 256 subvolumes a record
    n = 256 * records
    st = np.full((m.n_species, n), 4000, np.uint32)
    st[0, n - 1] = 9000  # its departures and decays bound the step
    with Simulation(m, seed=5) as sim:
        orc = Oracle.from_model(m, seed=5)
        sim.set_state(st.ravel())
        orc.set_state(st.ravel())
        for k in (1, 2, 1):  # fewer than the persistent kernel's three
            sim.step(k)
            orc.step(k)
            assert_same(sim, orc, f"{kind} {records} records")
