"""The full error matrix at the edges of its tiles and around the clip value,
where FP32 decides which pairs need FP64: equal to the oracle bit for bit."""
import numpy as np
import pytest

from abc_inference_transcription_gb300.config import REF_FAMILIES, make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,G,K", [(1, 1, 1), (63, 64, 16), (64, 65, 17), (65, 130, 53), (200, 3, 72), (129, 63, 300)])
def test_error_matrix_matches_oracle(built, orc, P, G, K):
    from abc_inference_transcription_gb300.host import Context
    rng = np.random.default_rng(P * 1000 + K)
    data = np.exp(rng.normal(0.0, 1.5, (G, K)))
    se = 0.1 * data * rng.lognormal(0.0, 0.5, (G, K))
    stats = np.exp(rng.normal(0.0, 1.5, (P, K)))
    # rows scaled so that their error for one gene is 10 but for a relative offset of 0 to 1e-3
    den = se * se + 0.01 * data * data
    for i in range(0, P, 2):
        g = i % G
        z = rng.normal(size=K)
        z *= np.sqrt(10.0 * K * (1.0 + rng.choice([0.0, 1e-15, -1e-15, 1e-9, -1e-9, 1e-6, -1e-6, 1e-4, -1e-4, 1e-3]))
                     / np.sum(z * z))
        stats[i] = data[g] - z * np.sqrt(den[g])
    special = [np.nan, np.inf, -np.inf, 1e39, -1e39, 1e-320, 1e200, 0.0]
    for j in range(min(P // 3, 40)):
        stats[3 * j, rng.integers(K)] = special[j % 8]
    for j in range(G // 4):
        data[4 * j, rng.integers(K)] = [0.0, 1e-200, 1e39, np.inf][j % 4]
        se[4 * j, rng.integers(K)] = [0.0, 1e-200, 1e39, 1e-45][j % 4]
    fam = list(REF_FAMILIES) if K == 53 else None
    with Context(make_config("hour"), None) as ctx:
        got = ctx.errors(data, se, stats, fam)
        again = ctx.errors(data[:1], se[:1], stats[:1], fam)
    want = orc.errors(data, se, stats, fam)
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(again, want[:1, :1], equal_nan=True)
