"""A call's workspace above the size that a context keeps (512 MB) is given back when
the call returns, whether with a result or with a refusal."""
import numpy as np
import pytest
import torch

from abc_inference_transcription_gb300.abi import AbcError
from abc_inference_transcription_gb300.config import make_config, synthetic_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [3, -1])
def test_large_workspace_is_given_back(built, count):
    from abc_inference_transcription_gb300.host import Context

    cells = synthetic_cells(n_per_pulse=10, n_per_chase=10, seed=2)
    u = np.full((300, cells.n), count, np.int32)
    with Context(make_config("hour"), cells) as ctx:
        ctx.data_stats(np.zeros_like(u), np.zeros_like(u), n_boot=2, seed=1)
        before = torch.cuda.mem_get_info()[0]
        n_boot = 10_000  # 53 statistics of 300 x 10,001 resamples: 1.3 GB
        if count < 0:
            with pytest.raises(AbcError, match="counts"):
                ctx.data_stats(u, u, n_boot=n_boot, seed=1)
        else:
            ctx.data_stats(u, u, n_boot=n_boot, seed=1)
        assert before - torch.cuda.mem_get_info()[0] < 600 << 20
