"""The production SSA's results do not depend on how its work is scheduled:
how many lanes of a warp take work, how many blocks per SM run, how long lanes
wait at a breakpoint together, and whether a lane or the warp halves a count."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from abc_inference_transcription_gb300 import abi
from abc_inference_transcription_gb300.config import make_config, synthetic_cells

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _thetas(rng, n):
    """From a few molecules to counts above the lane-halving limit."""
    th = np.tile(np.log10([0.5, 1.0, 20.0, 0.1, 0.7]), (n, 1))
    th[:, 2] = np.linspace(-1.0, 2.5, n)
    return th + rng.uniform(-0.2, 0.0, (n, 5))


@pytest.mark.parametrize("n,per_pulse,kw", [(2, 10, {}), (7, 20, {}), (40, 200, {}), (9, 20, {"splicing": True}),
                                            (9, 20, {"scaling_column": True}), (5, 20, {"ages": 0.3})])
def test_batch_equals_single_particles(built, n, per_pulse, kw):
    from abc_inference_transcription_gb300.host import Context
    ages = kw.get("ages")
    cfg = make_config("hour", precision=abi.FP32, splicing=kw.get("splicing", False),
                      scaling_column=kw.get("scaling_column", False))
    if ages:  # times off the power-of-two grid: breakpoints in FP64
        for a in range(cfg.n_ages):
            cfg.ages[a] += ages
    cells = synthetic_cells(n_per_pulse=per_pulse, n_per_chase=per_pulse, seed=4)
    rng = np.random.default_rng(n)
    theta = _thetas(rng, n)
    if kw.get("splicing"):
        theta = np.hstack([theta, np.full((n, 1), 0.3)])
    if kw.get("scaling_column"):
        theta = np.hstack([theta, np.full((n, 1), 0.8)])
    with Context(cfg, cells) as ctx:
        whole = ctx.simulate_cells(1, theta, seed=9)
        total = ctx.last_counters()
        single = [ctx.simulate_cells(1, theta[p:p + 1], seed=9, offset=p) for p in range(n)]
        for key in ("counts", "captured", "events"):
            assert np.array_equal(whole[key], np.concatenate([s[key] for s in single])), key
        assert whole["events"].sum() == total[0]
        for variant, chunk in ((1, 1), (0, 3)):
            ctx.set_variant(variant)
            ctx.set_work_chunk(chunk)
            other = ctx.simulate_cells(1, theta, seed=9)
            assert np.array_equal(whole["counts"], other["counts"]) and ctx.last_counters() == total


def test_lane_and_warp_halving_agree(built, tmp_path):
    so = tmp_path / "libhalve.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-shared", "-Xcompiler", "-fPIC", os.path.join(ROOT, "tests", "gpu_helpers", "halve.cu"), "-o",
                    str(so)], check=True)
    lib = C.CDLL(str(so))
    out = np.zeros((1200, 4), np.int32)
    for seed in (1, 2 ** 40 + 5):
        assert lib.halve_counts(C.c_ulonglong(seed), 1200, out.ctypes.data_as(C.POINTER(C.c_int))) == 0
        assert np.array_equal(out[:, 0], out[:, 1]) and np.array_equal(out[:, 2], out[:, 3])
        n = np.arange(1200)
        assert (np.abs(out[:, 0] - n / 2) <= 4 * np.sqrt(n) + 1).all() and (out[:, 0] <= n).all()


@pytest.mark.parametrize("n,n_steps,model,kw", [(1, 5, 1, {}), (3, 1, 4, {}), (4, 8, 3, {}), (5, 2, 5, {}),
                                                (7, 5, 2, {"splicing": True}), (6, 8, 5, {"scaling_column": True})])
def test_particle_records_match_oracle(built, orc, n, n_steps, model, kw):
    """Rates, initial moments and statistics of particle groups that do not fill
    a warp, for the smallest and largest numbers of age steps: the FP64 mode's
    counts equal the oracle's, with an invalid parameter set between them."""
    from abc_inference_transcription_gb300.host import Context
    cfg = make_config("hour", precision=abi.FP64, **kw)
    cfg.n_steps = n_steps
    cells = synthetic_cells(n_per_pulse=10, n_per_chase=10, seed=2)
    npar = abi.num_params(cfg, model)
    rng = np.random.default_rng(n)
    theta = rng.uniform(-1.0, 0.6, (n, npar))
    if cfg.scaling_column:  # a negative size exponent is refused
        theta[:, -1] = np.abs(theta[:, -1])
    with Context(cfg, cells) as ctx:
        got = ctx.simulate_cells(model, theta, seed=3)
        ref = orc.simulate(cfg, cells, model, theta, seed=3)
        for key in ("counts", "captured", "events", "hash"):
            assert np.array_equal(got[key], ref[key]), key
        assert np.array_equal(got["stats"], ref["stats"], equal_nan=True)
        if n > 2:
            bad = theta.copy()
            bad[1, 0] = np.nan
            with pytest.raises(abi.AbcError):
                ctx.simulate(model, bad, seed=3)
            assert np.array_equal(ctx.simulate(model, theta, seed=3), got["stats"], equal_nan=True)
