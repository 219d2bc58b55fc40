"""Top-q selections whose threshold, taken from a strided subsample, is too narrow:
the subsample sees none but particles near the genes, so the candidate pass runs
again with wider thresholds, and once more where those do not do either."""
import numpy as np
import pytest

from abc_inference_transcription_gb300.config import make_config

pytestmark = pytest.mark.gpu

SUB = 32768  # particles of the subsample


@pytest.mark.parametrize("mode", (0, 1, 2, 3))
@pytest.mark.parametrize("far,passes", ((0.05, 2), (0.3, 3)))
@pytest.mark.parametrize("errors", (True, False))
def test_thresholds_widened(built, orc, mode, far, passes, errors):
    from abc_inference_transcription_gb300.host import Context

    P, G, K = 4 * SUB, 5, 8
    rng = np.random.default_rng(3)
    data = rng.lognormal(1.0, 0.3, (G, K))
    data[1:3] = data[0] * 1.01  # genes whose threshold is too narrow, and two far from everything
    data[3:] *= 50.0
    se = 0.1 * data
    stats = data[0] * (1.0 + far * rng.choice((-1.0, 1.0), (P, K)) * rng.uniform(0.9, 1.1, (P, K)))
    stats[::4] = data[0] * (1.0 + 0.02 * rng.normal(size=(SUB, K)))
    with Context(make_config("hour"), None) as ctx:
        ctx.set_distance_mode(mode)
        off, idx, err = ctx.select(data, se, stats, 1, 0.3, None, errors=errors)
        cands = ctx.select_counters()[0]
    full = orc.errors(data, se, stats, None)
    want_off, want_idx = orc.accept(full, 1, 0.3)
    assert np.array_equal(off, want_off) and np.array_equal(idx, want_idx)
    if errors:
        assert np.array_equal(err, full[idx - 1, np.repeat(np.arange(G), np.diff(off))])
    assert cands >= passes * 2 * P  # two genes' errors are all clipped: every pass finds all their pairs
