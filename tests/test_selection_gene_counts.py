"""Selections at the gene counts where the selection's kernels change: 16-gene
tiles up to 32 genes, candidate histograms in shared memory up to 12, 1 to 8
genes per threshold CTA from 304 on (with a last CTA that is not full), and
rechecks of fewer pairs than fill one warp per block."""
import numpy as np
import pytest

from abc_inference_transcription_gb300.config import REF_FAMILIES, make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [1, 4, 12, 13, 16, 17, 32, 33, 303, 305, 1217])
def test_selection_matches_oracle(built, orc, G):
    from abc_inference_transcription_gb300.host import Context

    K, P = sum(REF_FAMILIES), 3001
    rng = np.random.default_rng(500 + G)
    base = np.abs(rng.normal(5.0, 3.0, (300, K))) + 0.1
    stats = base[rng.integers(0, 300, P)] * rng.lognormal(0, 0.2, (P, K))
    stats[17] = np.nan
    stats[40:45] = stats[39]  # exact ties, broken by index
    data = base[rng.integers(0, 300, G)] * rng.lognormal(0, 0.05, (G, K))
    se = 0.1 * np.abs(data) * rng.lognormal(0, 0.5, (G, K))
    err = orc.errors(data, se, stats, REF_FAMILIES)
    with Context(make_config("hour"), None) as ctx:
        for sel, x in ((0, 4.8), (1, 0.0004), (1, 0.05)):
            off, idx, e = ctx.select(data, se, stats, sel, x, REF_FAMILIES)
            roff, ridx = orc.accept(err, sel, x)
            assert np.array_equal(off, roff) and np.array_equal(idx, ridx), (sel, x)
            genes = np.repeat(np.arange(G), np.diff(off))
            assert np.array_equal(e, err[idx - 1, genes])
