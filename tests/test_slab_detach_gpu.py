"""A proposer detached from the handles of z-slabs (a call that changes nothing there): the slabs stay whole
bricks on a lattice that a single domain cuts into runs, and follow the single domain bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_slabs_stay_bricks_when_a_proposer_is_detached(precision, monkeypatch):
    import test_slabs_gpu
    from pliscuda_b200 import slabs
    from test_runs_gpu import _schlogl

    class Detached(slabs.Slab):
        def __init__(self, *a, **kw):
            super().__init__(*a, **kw)
            self.sim.set_proposer(None)

    monkeypatch.setattr(slabs, "Slab", Detached)
    m, st = _schlogl((19, 21, 18))
    assert test_slabs_gpu._compare(m, st, [(0, 8), (8, 18)], 0.02, seed=5, precision=precision).steps > 3
