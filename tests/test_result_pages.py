"""Results of top-q selections allocated before the selection (2^18 pairs and
more) are those of the same genes selected one by one, whose results are
allocated after it; with fewer errors than q asks for, the result is shorter
than the named arrays."""
import ctypes as C
import math

import numpy as np
import pytest

from abc_inference_transcription_gb300.abi import ptr
from abc_inference_transcription_gb300.config import REF_FAMILIES, make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("errors", [True, False])
@pytest.mark.parametrize("G,q,nan", [(53, 0.1, 0.0), (52, 0.1, 0.0), (64, 0.2, 0.9)])
def test_topq_results_allocated_beforehand(built, G, q, nan, errors):
    from abc_inference_transcription_gb300.host import Context

    K, P = sum(REF_FAMILIES), 50001
    rng = np.random.default_rng(G)
    stats = rng.lognormal(1.0, 0.5, (P, K))
    stats[rng.permutation(P)[:int(nan * P)]] = np.nan
    data = rng.lognormal(1.0, 0.3, (G, K))
    se = 0.1 * data
    k = math.ceil(q * P)
    assert (G * k >= Context._OWN_MIN) == (G != 52)
    with Context(make_config("hour"), None) as ctx:
        off, idx, err = ctx.select(data, se, stats, 1, q, REF_FAMILIES, errors=errors)
        assert idx.shape[0] == off[-1] and (err is None) == (not errors)
        assert (off[-1] == G * k) == (nan < 1.0 - q)
        for g in (0, G // 2, G - 1):
            o1, i1, e1 = ctx.select(data[g:g + 1], se[g:g + 1], stats, 1, q, REF_FAMILIES, errors=errors)
            assert np.array_equal(idx[off[g]:off[g + 1]], i1)
            if errors:
                assert np.array_equal(err[off[g]:off[g + 1]], e1)


def test_named_output_is_left_as_it_is(built):
    """The pages are made present, odd ends of the array included; its contents
    and a selection that returns less than was named stay what they were."""
    from abc_inference_transcription_gb300.host import Context

    K = sum(REF_FAMILIES)
    rng = np.random.default_rng(2)
    stats, data = rng.lognormal(1.0, 0.5, (3001, K)), rng.lognormal(1.0, 0.3, (3, K))
    room = np.full((1 << 20) + 7, -5, np.int64)
    with Context(make_config("hour"), None) as ctx:
        want = ctx.select(data, 0.1 * data, stats, 1, 0.01, REF_FAMILIES)
        part = room[3:-3]
        assert ctx.lib.abc_select_output(ctx.h, ptr(part, C.c_int64), None, part.shape[0]) == 0
        got = ctx.select(data, 0.1 * data, stats, 1, 0.01, REF_FAMILIES)
        assert all(np.array_equal(a, b) for a, b in zip(want, got))
        assert (room == -5).all()
        assert ctx.lib.abc_select_output(ctx.h, ptr(part, C.c_int64), None, -1) != 0
