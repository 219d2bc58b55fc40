"""Posterior summaries and model probabilities at the list lengths and counts where
their kernels change: order statistics of 2 values and around the sizes that are
ranked by counting (64) and staged in shared memory (2,048), loads ahead of the
mean's chain (8); resamples below, at and above a thread's first, and totals at
the ends of a radix digit."""
import numpy as np
import pytest

from abc_inference_transcription_gb300.config import make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 7, 8, 9, 63, 64, 65, 2047, 2048, 2049])
def test_summary_of_k_accepted(built, orc, k):
    from abc_inference_transcription_gb300.host import Context

    rng = np.random.default_rng(k)
    K, G, P = 6, 5, 4100
    stats = np.abs(rng.normal(5.0, 1.0, (P, K))) + 0.1
    data = stats[rng.integers(0, P, G)] * 1.01
    theta = rng.normal(size=(P, 3))
    theta[:, 1] = np.round(theta[:, 1])  # ties
    theta[:, 2] = 0.25                   # one value
    with Context(make_config("hour"), None) as ctx:
        off, idx, _ = ctx.select(data, 0.1 * data, stats, 1, (k + 0.5) / P, None)
        got = ctx.posterior_summary(theta, q=0.9)
    assert (np.diff(off) >= k).all()
    want = orc.posterior_summary(theta, off, idx, 0.9)
    for name in ("map", "mean", "lower", "upper", "n_particles"):
        assert np.array_equal(got[name], want[name], equal_nan=True), name


@pytest.mark.parametrize("n_boot", [1, 2, 64, 65, 257])
def test_model_probs_of_small_and_large_totals(built, orc, n_boot):
    from abc_inference_transcription_gb300.host import Context

    counts = np.array([[1, 1, 0], [100, 100, 55], [100, 100, 56], [60000, 5000, 535], [60000, 5000, 536],
                       [1, 2 ** 24, 7], [3, 2 ** 33, 2 ** 33], [0, 5, 0]], np.int64)
    with Context(make_config("hour"), None) as ctx:
        got = ctx.model_probs(counts, n_boot=n_boot, alpha=0.9, seed=3)
    for a, b in zip(got, orc.model_probs(counts, n_boot=n_boot, alpha=0.9, seed=3)):
        assert np.array_equal(a, b)
