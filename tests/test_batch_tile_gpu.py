"""A batch keeps the bricks of a tile that its caller gives, the default's shape included.  9 x 9 x 9 replicas take
twelve bricks of 8 x 8 x 4, a third full at most, and three runs of 256 by default: the same results, and four times the
work-queue entries cost the explicit bricks more device time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_explicit_default_shape_keeps_bricks():
    from pliscuda_b200 import workloads
    from pliscuda_b200.batch import Batch
    m, st = workloads.schlogl(9)
    n = 512

    def ms(b):
        best = 1e30
        for _ in range(4):
            for r in range(n):
                b.set_state(r, st)
            t0 = b.stats(0).device_ms
            b.step(40)
            best = min(best, b.stats(0).device_ms - t0)
        return best

    with Batch.from_models([m] * n, seed=4) as runs, Batch.from_models([m] * n, seed=4, tile=(8, 8, 4)) as bricks:
        t_runs, t_bricks = ms(runs), ms(bricks)
        assert bricks.tuning()["tile"] == runs.tuning()["tile"] == (8, 8, 4)
        for r in (0, 255, 511):
            assert np.array_equal(runs.get_state(r), bricks.get_state(r))
        assert t_bricks > 1.1 * t_runs, (t_bricks, t_runs)
        # the autotuner's 8 x 8 x 4 is the default cut again; whatever it picks, the results stay
        bricks.autotune(2)
        bricks.step(3)
        runs.step(3)
        assert np.array_equal(runs.get_state(7), bricks.get_state(7))
