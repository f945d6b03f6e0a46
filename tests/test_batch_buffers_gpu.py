"""A batch's states from pageable and from pinned buffers that the caller reuses at once, on both sides of the 64 KB
from which the driver copies a pageable buffer in parts: exact copies, and every replica steps from its own state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("side", [7, 25, 26, 60])
def test_buffers_reused_at_once(side, pinned):
    import torch
    from pliscuda_b200 import workloads
    from pliscuda_b200.batch import Batch
    m, _ = workloads.brusselator(side, 100.0, 300.0)
    n = m.n_subvolumes
    rng = np.random.default_rng(side)
    states = [np.concatenate([rng.poisson(100, n), rng.poisson(30000, n)]).astype(np.uint32) for _ in range(9)]
    buf = torch.empty(2 * n, dtype=torch.int32, pin_memory=pinned).numpy().view(np.uint32)
    with Batch.from_models([m] * len(states), seed=3) as b, Batch.from_models([m] * len(states), seed=3) as ref:
        for r, st in enumerate(states):
            buf[:] = st
            b.set_state(r, buf)
            buf[:] = 1
            ref.set_state(r, st)
        for r, st in enumerate(states):
            assert np.array_equal(b.get_state(r), st)
        b.step(3)
        ref.step(3)
        for r in range(len(states)):
            assert np.array_equal(b.get_state(r), ref.get_state(r))
