"""Top-q selections whose cut lies at the clip value, where ties are ordered by
index: the candidates kept for the recheck must hold the lowest indices of the ties
wherever the errors below the clip value, those barely above it and the particles
without an error lie among them."""
import numpy as np
import pytest

from abc_inference_transcription_gb300.config import make_config

pytestmark = pytest.mark.gpu

P, K = 50021, 8


def _stats(rng, data, order):
    """A tenth of the particles near the first gene, a tenth with errors of 10 but for a
    relative offset of up to 1e-6 either way, three tenths without an error, the rest far off."""
    n = P // 10
    z = rng.normal(size=(P, K))
    z /= np.sqrt((z * z).mean(axis=1, keepdims=True))  # mean square 1: the error is the square of the scale
    scale = np.full(P, 40.0)
    kind = np.repeat(np.arange(4), [n, n, 3 * n, P - 5 * n])
    kind = {"mixed": rng.permutation(kind), "near first": kind, "near last": kind[::-1],
            "none first": np.roll(kind, -2 * n), "border first": np.roll(kind, -n)}[order]
    scale[kind == 0] = rng.uniform(0.3, 3.0, n)
    scale[kind == 1] = np.sqrt(10.0) * (1.0 + rng.uniform(-1e-6, 1e-6, n))
    stats = data[0] + z * scale[:, None] * np.sqrt(2.0) * 0.1 * data[0]
    stats[kind == 2] = np.nan
    return stats


@pytest.mark.parametrize("mode", (0, 1, 2, 3))
@pytest.mark.parametrize("G", (2, 14))  # histograms of the candidates in shared and in global memory
@pytest.mark.parametrize("order", ("mixed", "near first", "near last", "none first", "border first"))
def test_cut_at_the_clip_value(built, orc, mode, G, order):
    from abc_inference_transcription_gb300.host import Context

    rng = np.random.default_rng(7)
    data = rng.lognormal(1.0, 0.3, (G, K))
    data[1:] = data[0] * (1.0 + 0.2 * np.arange(1, G)[:, None])
    stats = _stats(rng, data, order)
    se = 0.1 * data
    full = orc.errors(data, se, stats, None)
    with Context(make_config("hour"), None) as ctx:
        ctx.set_distance_mode(mode)
        # a cut below the clip value, within the errors around it, among the ties, and beyond the last error
        for q in (0.05, 0.15, 0.21, 0.5, 0.6995, 0.71):
            want_off, want_idx = orc.accept(full, 1, q)
            for errors in (True, False):
                off, idx, err = ctx.select(data, se, stats, 1, q, None, errors=errors)
                assert np.array_equal(off, want_off) and np.array_equal(idx, want_idx), (q, errors)
                if errors:
                    assert np.array_equal(err, full[idx - 1, np.repeat(np.arange(G), np.diff(off))])
