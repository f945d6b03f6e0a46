"""A proposer with the clamp 1 (the plain method) on the handles of z-slabs: the decisions are taken for a slab's
own subvolumes only, whatever the device memory held before, and the slabs follow the single domain bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


def _dirty_device_memory():
    """Device memory that the next small allocations get, full of twos."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    blocks = []
    for size in (4096, 65536, 1 << 20):
        for _ in range(64):
            err, p = rt.cudaMalloc(size)
            assert int(err) == 0
            rt.cudaMemset(p, 2, size)
            blocks.append(p)
    rt.cudaDeviceSynchronize()
    for p in blocks:
        rt.cudaFree(p)


@pytest.mark.parametrize("bounds", [[(0, 8), (8, 16)], [(0, 4), (4, 16)]], ids=["halves", "uneven"])
def test_slabs_decide_their_own_subvolumes(bounds, monkeypatch):
    import test_slabs_gpu
    from pliscuda_b200 import slabs, workloads
    from test_learned_gpu import random_weights

    class Learned(slabs.Slab):
        def __init__(self, *a, **kw):
            _dirty_device_memory()
            super().__init__(*a, **kw)
            self.sim.set_proposer(random_weights(3), 1.0)

    monkeypatch.setattr(slabs, "Slab", Learned)
    m, st = workloads.schlogl(16)
    assert test_slabs_gpu._compare(m, st, bounds, 0.05, seed=21, mode=1).steps > 20
