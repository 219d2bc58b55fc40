"""Arrays named for the next selection's result belong to that call alone, also
where it is refused: a later selection must not touch their pages."""
import ctypes as C
import mmap

import numpy as np
import pytest

from abc_inference_transcription_gb300 import abi
from abc_inference_transcription_gb300.abi import ptr
from abc_inference_transcription_gb300.config import REF_FAMILIES, make_config

pytestmark = pytest.mark.gpu

LIBC = C.CDLL(None, use_errno=True)


def _resident(address, size):
    pages = (C.c_ubyte * (size // mmap.PAGESIZE))()
    assert LIBC.mincore(C.c_void_p(address), C.c_size_t(size), pages) == 0
    return sum(p & 1 for p in pages)


@pytest.mark.parametrize("call", ["mode", "genes", "null"])
def test_refused_selection_forgets_the_named_arrays(built, call):
    from abc_inference_transcription_gb300.host import Context

    K, P, size = sum(REF_FAMILIES), 2000, 4 << 20
    rng = np.random.default_rng(1)
    stats, data = rng.lognormal(1.0, 0.5, (P, K)), rng.lognormal(1.0, 0.3, (3, K))
    se = 0.1 * data
    tot = C.c_int64()
    room = mmap.mmap(-1, size)
    first = (C.c_char * size).from_buffer(room)
    address = C.addressof(first)
    with Context(make_config("hour"), None) as ctx:
        assert ctx.lib.abc_select_output(ctx.h, C.cast(address, C.POINTER(C.c_int64)), None, size // 8) == 0
        G, mode, d = (3, 2, ptr(data)) if call == "mode" else (0, 1, ptr(data)) if call == "genes" else (3, 1, None)
        st = ctx.lib.abc_errors_select(ctx.h, d, ptr(se), G, K, 0, None, ptr(stats), P, mode, 0.01, C.byref(tot))
        assert st == abi.ERR_INVALID
        ctx.select(data, se, stats, 1, 0.01, REF_FAMILIES)
        assert _resident(address, size) == 0
