"""The full error matrix with every number of particles per tile (4 to 32, by the
matrix's size), genes split evenly or not, last tiles partly empty: none, half and
all of the pairs below the clip value, equal to the oracle bit for bit."""
import numpy as np
import pytest

from abc_inference_transcription_gb300.config import make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,G", [(3, 1), (61, 65), (607, 100), (1201, 130), (2431, 2), (2433, 5), (4849, 3), (4867, 64),
                                 (9697, 1), (9729, 2), (3203, 193)])
@pytest.mark.parametrize("near", [0.0, 0.5, 1.0])
def test_tiles(built, orc, P, G, near):
    from abc_inference_transcription_gb300.host import Context

    K = 9
    rng = np.random.default_rng(P + G)
    data = np.exp(rng.normal(0.0, 0.02, (G, K))) * np.exp(rng.normal(0.0, 1.0, K))
    se = 0.1 * data
    stats = data[0] * np.exp(rng.normal(0.0, 0.05, (P, K)))
    far = rng.random(P) >= near
    stats[far] *= 30.0
    with Context(make_config("hour"), None) as ctx:
        got = ctx.errors(data, se, stats, None)
    want = orc.errors(data, se, stats, None)
    assert np.array_equal(got, want)
    assert (want[far] == 10.0).all() and (want[~far] < 10.0).all()
