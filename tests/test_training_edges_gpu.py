"""The training kernel (k_train in pliscuda_b200/csrc/learned.cu) where a CTA's 128 records do not fill or
are unusable: the gradient against a float64 backward pass, with the tolerance of the gradient test of
1,000 records (sums of at most 1,024 binary32 products)."""
import numpy as np
import pytest

from test_learned_gpu import _learner, loss_grad_f64, random_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,unusable", [(1, 0), (31, 3), (127, 0), (128, 40), (129, 0), (513, 100)])
def test_gradient_of_partial_blocks(n, unusable):
    from pliscuda_b200.learned import TRACE_DTYPE
    rng = np.random.default_rng(n)
    recs = np.zeros(n, TRACE_DTYPE)
    recs["features"] = rng.normal(0, 2, (n, 8))
    recs["label"] = rng.normal(0.5, 1.0, n)
    recs["tau_cao"] = 1.0
    bad = rng.permutation(n)[:unusable]
    recs["label"][bad] = np.nan
    w = random_weights(2)
    with _learner() as L:
        L.set_weights(w)
        L.set_records(recs)
        g, loss = L.gradient(0.25)
    good = np.delete(np.arange(n), bad)
    lref, gref = loss_grad_f64(w, recs["features"][good], recs["label"][good].astype(np.float64), 0.25)
    lref, gref = lref * len(good) / n, gref * len(good) / n  # the means run over all records
    assert abs(loss - lref) < 1e-4 * (1 + abs(lref))
    err = np.abs(g - gref) / (np.abs(gref).max() + 1e-30)
    assert err.max() < 1e-4, err.max()


def test_training_is_deterministic_and_odd_batches_work():
    from pliscuda_b200.learned import TRACE_DTYPE
    rng = np.random.default_rng(9)
    recs = np.zeros(1000, TRACE_DTYPE)
    recs["features"] = rng.normal(0, 2, (1000, 8))
    recs["label"] = rng.normal(0.5, 1.0, 1000)
    recs["tau_cao"] = 1.0
    for batch in (128, 384):
        runs = []
        for _ in range(2):
            with _learner() as L:
                L.set_records(recs)
                rep = L.train(iterations=40, batch=batch, seed=5)
                runs.append((L.weights(), rep["loss_last"]))
        assert np.array_equal(runs[0][0], runs[1][0]) and runs[0][1] == runs[1][1]
        assert np.isfinite(runs[0][0]).all()
