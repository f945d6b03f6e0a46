"""State transfers through the pinned slices (pliscuda_b200/csrc/host_stage.h): sizes around one slice, around
the limits of the threaded path and with ragged last parts, several rows, pageable and pinned buffers,
buffers reused at once, and refused states that leave the old one in place.  Exact: copies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sim(n, species):
    from pliscuda_b200 import Simulation, workloads
    m = workloads._model((n, 1, 1), species, [({}, {0: 1})], [0.0], [0.0] * species)
    return Simulation(m)


@pytest.mark.parametrize("n,species", [(1, 1), (1000, 3), ((1 << 21) + 33, 1), ((1 << 23) - 1, 1), (1 << 23, 1), ((1 << 23) + 33, 1),
                                       (700_001, 13), (524_289, 17)])
def test_round_trip(n, species):
    import torch
    rng = np.random.default_rng(n)
    with _sim(n, species) as sim:
        for k in range(2):
            c = rng.integers(0, 1 << 30, size=n * species, dtype=np.uint32)
            keep = c.copy()
            sim.set_state(c)
            c[:] = 7  # the caller's buffer is free once the call has returned
            assert np.array_equal(sim.get_state(), keep)
        pinned = torch.empty(n * species, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
        pinned[:] = keep[::-1]
        sim.set_state(pinned)
        out = torch.empty(n * species, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
        assert np.array_equal(sim.get_state(out), keep[::-1]) and np.array_equal(sim.get_state(), keep[::-1])


@pytest.mark.parametrize("n", [100, (1 << 23) + 5])
def test_refused_state_leaves_the_old_one(n):
    from pliscuda_b200 import PlisError
    rng = np.random.default_rng(1)
    with _sim(n, 1) as sim:
        good = rng.integers(0, 1 << 30, size=n, dtype=np.uint32)
        sim.set_state(good)
        for place in (0, n // 2, n - 1):
            bad = good.copy()
            bad[place] = 1 << 30
            with pytest.raises(PlisError):
                sim.set_state(bad)
            assert np.array_equal(sim.get_state(), good)


def test_batch_states():
    """More replicas than slices, set and read in any order, before and after steps."""
    from pliscuda_b200 import workloads
    from pliscuda_b200.batch import Batch
    reps = [(m, st) for m, st, _ in workloads.brusselator_batch(21, side_range=(3, 12))]
    with Batch.from_models([m for m, _ in reps], seed=2) as b:
        order = np.random.default_rng(0).permutation(21)
        for r in order:
            c = reps[r][1].copy()
            b.set_state(int(r), c)
            c[:] = 0
        for r in order[::-1]:
            assert np.array_equal(b.get_state(int(r)), reps[r][1])
        b.step(3)
        first = [b.get_state(r) for r in range(21)]
        assert all(b.stats(r).steps == 3 for r in range(21))
        b.set_state(4, reps[4][1])
        assert b.stats(4).steps == 0 and np.array_equal(b.get_state(4), reps[4][1])
        assert all(np.array_equal(b.get_state(r), first[r]) for r in range(21) if r != 4)
        for r in range(21):
            b.set_state(r, reps[r][1])
        b.step(3)
        assert all(np.array_equal(b.get_state(r), first[r]) for r in range(21))
