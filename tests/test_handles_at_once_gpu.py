"""Several handles stepped by threads of their own at the same time: systems in the persistent step kernel (cooperative
launches on different streams) and in phase kernels side by side give what each gives alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_with_handles_of_their_own():
    from pliscuda_b200 import Simulation, workloads
    from helpers import birth_death_model
    systems = [workloads.small_ab(10, seed=3), workloads.schlogl(16), workloads.schlogl(24), birth_death_model(12),
               workloads.schlogl(48), workloads.small_ab(10, seed=3)]

    def single(i, out):
        m, st = systems[i]
        with Simulation(m, seed=9, replica=i, mode=i % 2) as sim:
            got = []
            for n in (40, 3, 1, 60):
                sim.set_state(st)
                sim.step(n)
                got.append((sim.get_state(), sim.stats().time, sim.stats().events))
            out[i] = got

    jobs = range(len(systems))
    alone, together = {}, {}
    for i in jobs:
        single(i, alone)
    for _ in range(3):
        together.clear()
        threads = [threading.Thread(target=single, args=(i, together)) for i in jobs]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i in jobs:
            for a, b in zip(alone[i], together[i], strict=True):
                assert np.array_equal(a[0], b[0]) and a[1:] == b[1:], f"system {i}"
