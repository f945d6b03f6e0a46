"""plis_tau_argmin_noalloc at the edges of its paths: one CTA or two passes, 16-byte loads with an
unaligned first element and an odd last one, unrolled rounds and remainders; the minimum first, last
and in between, ties, and NaNs.  A min: the result is exact."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEP = 888 * 256  # double2 per round of the largest grid


@pytest.mark.parametrize("n", [1, 2, 3, 511, 512, 513, 8191, 8192, 8193, 8194, 65_537, 2 * STEP + 1, 16 * STEP - 1, 16 * STEP,
                               16 * STEP + 3, 40 * STEP + 5])
@pytest.mark.parametrize("offset", [0, 1])
def test_sizes_alignments_and_places(n, offset):
    import torch

    from pliscuda_b200 import _lib
    stream = torch.cuda.current_stream().cuda_stream
    base = torch.empty(n + offset, dtype=torch.float64, device="cuda")
    tau = base[offset:]
    assert base.data_ptr() % 16 == 0 and tau.data_ptr() % 16 == 8 * offset
    out_t = torch.empty(1, dtype=torch.float64, device="cuda")
    out_i = torch.empty(1, dtype=torch.int64, device="cuda")
    rng = np.random.default_rng(n)
    for places in ([0], [n - 1], [n // 2], sorted(int(v) for v in rng.integers(n, size=3)), []):
        base.fill_(2.0)
        if n > 4:
            tau[n // 3] = float("nan")
        for p in places:
            tau[p] = 1.0
        want = (1.0, places[0]) if places else (2.0, 0)
        rc = _lib.lib.plis_tau_argmin_noalloc(ctypes.c_void_p(tau.data_ptr()), n, ctypes.c_void_p(out_t.data_ptr()),
                                              ctypes.c_void_p(out_i.data_ptr()), ctypes.c_void_p(stream))
        assert rc == 0
        assert (out_t.item(), out_i.item()) == want, (places, n, offset)
