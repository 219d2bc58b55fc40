"""Moment simulation of batches with invalid particles, whole groups of neighbours
and single ones: their rows are NaN, the call says so, every other row is that of a
batch of valid particles, bit for bit, and the context goes on working."""
import numpy as np
import pytest

from abc_inference_transcription_gb300 import abi
from abc_inference_transcription_gb300.abi import ptr
from abc_inference_transcription_gb300.config import beta_moments, make_config, reference_prior, synthetic_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.FP32, abi.FP64])
@pytest.mark.parametrize("model", [1, 4])
def test_invalid_particles(built, precision, model):
    from abc_inference_transcription_gb300.host import Context

    cells = synthetic_cells(seed=2)
    bm = np.ascontiguousarray(beta_moments(cells, 5), np.float64)
    ad = np.ascontiguousarray(cells.age_dist, np.float64)
    iv = np.zeros(9)
    iv[1] = 0.5
    with Context(make_config("hour", precision=precision), cells) as ctx:
        theta = ctx.sample_prior(model, 33, 5, reference_prior())
        want = ctx.moment_simulate(model, theta, iv, bm, ad)["stats"]
        # a lone particle, the last one of a group of its own, whole groups of 8 among valid ones, all
        for n, bad in ((1, range(1)), (9, range(8, 9)), (16, range(0, 8)), (16, range(8, 16)), (33, range(8, 25)),
                       (33, range(33)), (33, (0, 31, 32))):
            for value in (np.nan, 400.0):  # not a number; a rate beyond the FP64 range
                th = theta[:n].copy()
                th[list(bad), 0] = value
                got = np.full((n, ctx.K), -1.0)
                st = ctx.lib.abc_moment_simulate(ctx.h, model, ptr(th), n, ptr(iv), 0.0, ptr(bm), 6, ptr(ad), ptr(got),
                                                 None, None)
                assert st == abi.ERR_NONFINITE, (n, bad, value)
                ok = np.ones(n, bool)
                ok[list(bad)] = False
                assert np.isnan(got[~ok]).all() and np.array_equal(got[ok], want[:n][ok], equal_nan=True)
        again = ctx.moment_simulate(model, theta, iv, bm, ad)["stats"]
        assert np.array_equal(again, want, equal_nan=True)
