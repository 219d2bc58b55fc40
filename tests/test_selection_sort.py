"""The per-gene sort at the list lengths where its path changes: counting over
the whole list up to 256 entries, one window of bins up to 8,192, several
windows above; the bitonic networks for crowded bins (one far entry, or exact
ties); ties at the clip value, binned by index.  eps = 10 accepts every
particle, so that a list is as long as the particles are many."""
import numpy as np
import pytest

from abc_inference_transcription_gb300.config import REF_FAMILIES, make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["spread", "crowded", "ties", "clipped", "all clipped"])
@pytest.mark.parametrize("n", [1, 2, 33, 255, 256, 257, 511, 512, 513, 4097, 8191, 8192, 8193, 16385, 40001])
def test_lists_of_every_length(built, orc, n, shape):
    from abc_inference_transcription_gb300.host import Context

    K = sum(REF_FAMILIES)
    rng = np.random.default_rng([n, len(shape)])
    base = rng.lognormal(1.0, 0.5, K)
    data = base * np.array([[1.0], [1.02]])
    se = 0.1 * data  # weights 50 / d^2: an error below 10 for deviations below 0.4 d
    far = rng.uniform(0.0, 0.35, (n, 1))
    if shape == "crowded":
        far = 1e-4 * far
        far[0] = 0.35
    stats = base * (1.0 + far * rng.uniform(-1.0, 1.0, (n, K)))
    if shape in ("clipped", "all clipped"):
        stats[rng.random(n) < (0.9 if shape == "clipped" else 1.1)] *= 3.0
    if shape == "ties":
        stats = stats[rng.integers(0, min(n, 7), n)]
    if n > 40:
        stats[5] = np.nan
    err = orc.errors(data, se, stats, REF_FAMILIES)
    with Context(make_config("hour"), None) as ctx:
        for errors in (True, False):
            for sel, x in ((0, 10.0), (1, 0.5)):
                off, idx, e = ctx.select(data, se, stats, sel, x, REF_FAMILIES, errors=errors)
                roff, ridx = orc.accept(err, sel, x)
                assert np.array_equal(off, roff) and np.array_equal(idx, ridx), (sel, errors)
                if errors:
                    assert np.array_equal(e, err[idx - 1, np.repeat(np.arange(2), np.diff(off))])
