"""Rank in a pool that takes long sessions: steps of short sessions alone, of long
ones alone and of both, with the step's stocks on both sides of the length where
the launches part; each session equal to its StreamContext run alone."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from kunquant_gb300 import serve
from tests.parity import compare_exact
from tests.test_gpu_serve import _alone, _data, _module


@pytest.mark.gpu
def test_short_and_long_sessions_of_a_large_pool():
    mod = _module("alpha101_stream")
    ex = kr.createSingleThreadExecutor()
    sizes = [64, 1, 1024, 5000, 1025, 900, 64]
    # which sessions each step takes: 64 to 8078 stocks
    steps = [[0], [0, 1, 6], [2], [4], [3], [0, 2, 5], [3, 4], [6, 3, 0], list(range(7)), [1, 5, 2, 6]] * 3
    ticks = [sum(i in s for s in steps) for i in range(len(sizes))]
    data = [_data(mod, S, T, seed=500 + i) for i, (S, T) in enumerate(zip(sizes, ticks))]
    want = [_alone(ex, mod, d) for d in data]
    pool = serve.ServePool(ex, mod, capacity_stocks=sum(sizes), max_sessions=40, max_session_stocks=16384,
                           start=False)
    sess = [pool.open(S) for S in sizes]
    clock = [0] * len(sizes)
    for step in steps:
        for i in step:
            for k in mod.getInputNames():
                sess[i].inputs[k][:] = data[i][k][clock[i]]
        pool.step([sess[i] for i in step])
        for i in step:
            got = {k: np.array(sess[i].outputs[k]) for k in mod.getOutputNames()}
            assert not compare_exact(got, {k: v[clock[i]] for k, v in want[i].items()}), (sizes[i], clock[i])
            clock[i] += 1
    pool.shutdown()


@pytest.mark.gpu
def test_a_pool_for_rows_that_rank_does_not_take_is_refused():
    mod = _module("alpha101_stream")
    pool = serve.ServePool(kr.createSingleThreadExecutor(), mod, capacity_stocks=64, max_sessions=4,
                           max_session_stocks=16385, start=False)
    with pytest.raises(kr.KunError):
        pool.step([pool.open(8)])
    pool.shutdown()
