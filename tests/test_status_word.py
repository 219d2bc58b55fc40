"""The status of stream-ordered simulations, read at synchronize, is theirs alone:
calls that check inputs of their own neither clear it nor add to it."""
import numpy as np
import pytest
import torch

from abc_inference_transcription_gb300.abi import AbcError
from abc_inference_transcription_gb300.config import beta_moments, make_config, reference_prior, synthetic_cells

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx(built):
    from abc_inference_transcription_gb300.host import Context
    with Context(make_config("hour"), synthetic_cells(n_per_pulse=10, n_per_chase=10, seed=2)) as c:
        yield c


def _simulate(ctx, theta):
    d_theta = torch.as_tensor(theta, device="cuda")
    d_stats = torch.empty((theta.shape[0], ctx.K), device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    ctx.simulate_device(1, d_theta.data_ptr(), theta.shape[0], 3, d_stats.data_ptr())
    return d_theta, d_stats


def _data_stats(ctx, count):
    u = np.full((3, ctx.cells.n), count, np.int32)
    ctx.data_stats(u, u, n_boot=10, seed=1)


def _moments(ctx, theta):
    iv = np.zeros(9)
    iv[1] = 0.5
    ctx.moment_simulate(1, theta, iv, beta_moments(ctx.cells, 5), ctx.cells.age_dist)


@pytest.mark.parametrize("call", ["data_stats", "moments"])
def test_status_of_a_simulation(ctx, call):
    theta = ctx.sample_prior(1, 4, 5, reference_prior()).clip(-1.0, 1.0)
    invalid = theta.copy()
    invalid[1, 0] = np.nan

    def between(ok):
        if call == "data_stats":
            _data_stats(ctx, 7 if ok else -1)
        else:
            _moments(ctx, theta if ok else invalid)

    # a failed simulation stays failed after a call that succeeds
    keep = _simulate(ctx, invalid)
    between(True)
    with pytest.raises(AbcError, match="non-finite"):
        ctx.synchronize()
    # a simulation that succeeds, or none, does not fail with a call that does
    keep = _simulate(ctx, theta)
    ctx.synchronize()
    with pytest.raises(AbcError):
        between(False)
    ctx.synchronize()
    keep = _simulate(ctx, theta)
    with pytest.raises(AbcError):
        between(False)
    ctx.synchronize()
    del keep
