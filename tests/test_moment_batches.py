"""FP32 moment simulation: a particle's results do not depend on the batch it is in,
bit for bit: batches that leave the kernels' particle tiles (4 to 128 threads)
partly empty, and one of more particles than a chunk of scratch holds."""
import numpy as np
import pytest

from abc_inference_transcription_gb300 import abi
from abc_inference_transcription_gb300.config import beta_moments, make_config, reference_prior, synthetic_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,h_max", [((1, 7, 8, 9, 31, 33, 127, 129), 0.0), ((1, 103, 104, 105), 20.0 / 8000)])
def test_results_do_not_depend_on_the_batch(built, sizes, h_max):
    from abc_inference_transcription_gb300.host import Context

    cells = synthetic_cells(seed=2)
    bm = beta_moments(cells, 5)
    iv = np.zeros(9)
    iv[1] = 0.5
    with Context(make_config("hour", precision=abi.FP32), cells) as ctx:
        theta = ctx.sample_prior(4, 2 * max(sizes), 41, reference_prior())

        def run(th):
            r = ctx.moment_simulate(4, th, iv, bm, cells.age_dist, moments=True, h_max=h_max)
            return r["stats"], r["moments"], r["transient_iters"]

        whole = run(theta)
        for n in sizes:
            for first in (0, theta.shape[0] - n):
                for got, want in zip(run(theta[first:first + n]), whole):
                    assert np.array_equal(got, want[first:first + n], equal_nan=True), (n, first)


@pytest.mark.parametrize("sizes,h_max", [((1, 2, 3, 4, 5, 127, 129), 0.0), ((1, 10), 20.0 / 8000)])
def test_exact_results_do_not_depend_on_the_batch(built, sizes, h_max):
    """The FP64 mode: three particles per warp of the walk, four of the paths, 128 of
    the exponentials; a chunk of scratch that holds fewer particles than the batch (55)."""
    from abc_inference_transcription_gb300.host import Context

    cells = synthetic_cells(seed=2)
    bm = beta_moments(cells, 5)
    iv = np.zeros(9)
    iv[1] = 0.5
    with Context(make_config("hour", precision=abi.FP64), cells) as ctx:
        theta = ctx.sample_prior(5, max(60, max(sizes) + 5), 43, reference_prior())

        def run(th):
            r = ctx.moment_simulate(5, th, iv, bm, cells.age_dist, moments=True, h_max=h_max)
            return r["stats"], r["moments"], r["transient_iters"]

        whole = run(theta)
        for n in sizes:
            for first in (0, theta.shape[0] - n):
                for got, want in zip(run(theta[first:first + n]), whole):
                    assert np.array_equal(got, want[first:first + n], equal_nan=True), (n, first)
