"""Handles destroyed in any order: a stream context or a serving pool keeps its
executor until it goes, as a program's end (which destroys objects in no
particular order) needs."""
import ctypes

import pytest

from kunquant_gb300 import runner as kr
from kunquant_gb300 import serve


@pytest.mark.gpu
def test_executor_destroyed_before_its_stream_and_pool():
    mod = kr.Library.predefined("alpha158_stream_f32").getModule("alpha158_stream")
    L = serve._lib()
    for first in (0, 1):
        ex = L.kunCreateMultiThreadExecutor(2)
        ctx = L.kunCreateStream(ex, mod.handle, 16)
        pool = ctypes.c_void_p()
        assert L.kunCreateServePool(ex, mod.handle, 64, 4, 32, ctypes.byref(pool)) == 0
        assert ex and ctx and pool.value
        L.kunDestoryExecutor(ex)
        for k in (first, 1 - first):
            if k:
                L.kunDestroyServePool(pool)
            else:
                L.kunDestoryStream(ctx)


@pytest.mark.gpu
def test_a_refused_stream_leaves_its_executor_usable():
    mod = kr.Library.predefined("alpha101_stream_f32").getModule("alpha101_stream")
    ex = kr.createSingleThreadExecutor()
    with pytest.raises(kr.KunError):
        kr.StreamContext(ex, mod, 16385)   # longer than Rank's rows: the tick is refused
    assert kr.StreamContext(ex, mod, 8).getCurrentBuffer(0).shape == (8,)
