"""Configurations in which one condition gives both the pulse and the chase
statistics (as the data side's may be): both families are written, and the same."""
import numpy as np
import pytest

from abc_inference_transcription_gb300 import abi
from abc_inference_transcription_gb300.config import beta_moments, make_config, reference_prior, synthetic_cells

A = 5


def _config(cond, precision=abi.FP64):
    cfg = make_config("hour", precision=precision)
    cfg.pulse_stat_cond = cfg.chase_stat_cond = cond
    return cfg


def _inputs(orc, cfg):
    cells = synthetic_cells(n_per_pulse=12, n_per_chase=12, seed=2)
    theta = orc.sample_prior(cfg, 1, 5, 3, reference_prior()).clip(-1.5, 1.0)
    iv = np.zeros(9)
    iv[1] = 0.5
    return cells, theta, iv, beta_moments(cells, A)


@pytest.mark.parametrize("cond", (0, 6, 10))
def test_oracle_writes_both(orc, cond):
    cfg = _config(cond)
    cells, theta, iv, bm = _inputs(orc, cfg)
    for th in theta:
        st = orc.moment_model(cfg, 1, th, iv, beta_mom=bm, age_dist=cells.age_dist)["stats"]
        assert np.array_equal(st[:2 * A], st[2 * A:4 * A])
        assert (st[:A] > 0.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("cond", (0, 6, 10))
def test_gpu_writes_both(built, orc, cond):
    from abc_inference_transcription_gb300.host import Context

    cfg = _config(cond)
    cells, theta, iv, bm = _inputs(orc, cfg)
    with Context(cfg, cells) as ctx:
        mom = ctx.moment_simulate(1, theta, iv, bm, cells.age_dist)["stats"]
        sim = ctx.simulate(1, theta, 7)
    want = [orc.moment_model(cfg, 1, th, iv, beta_mom=bm, age_dist=cells.age_dist)["stats"] for th in theta]
    assert np.array_equal(mom, want, equal_nan=True)
    with Context(_config(cond, abi.FP32), cells) as ctx:
        fast = ctx.moment_simulate(1, theta, iv, bm, cells.age_dist)["stats"]
        fast_sim = ctx.simulate(1, theta, 7)
    for st in (sim, fast, fast_sim):
        assert np.array_equal(st[:, :2 * A], st[:, 2 * A:4 * A], equal_nan=True)
        assert (st[:, :A] >= 0.0).all()
