"""Runs whose kernels are ordered by what they read (executors of several
streams) against the stage-by-stage run of a single stream: the same bits, on
first and replayed runs, with the arena's slots shared by more kernels, for one
universe and for many."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from kunquant_gb300 import synth
from tests.parity import compare_exact


def _dev(data):
    import torch
    return {k: torch.from_numpy(v).cuda() for k, v in data.items()}


def _cpu(out):
    return {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.gpu
@pytest.mark.parametrize("key,name", [("alpha101_f32", "alpha101"), ("alpha158_f32", "alpha158"),
                                      ("alpha158_f64", "alpha158_f64"), ("alpha158_slide_f32", "alpha158_slide")])
@pytest.mark.parametrize("S,T,start", [(1, 70, 0), (37, 263, 20), (1100, 300, 0)])
def test_streams_do_not_change_results(key, name, S, T, start):
    dt = np.float64 if key.endswith("f64") else np.float32
    mod = kr.Library.predefined(key).getModule(name)
    data = synth.ohlcv(S, T, seed=S + T, nan_frac=0.01, dtype=dt)
    want = _cpu(kr.runGraph(kr.createSingleThreadExecutor(), mod, _dev(data), start, T - start))
    for streams in (2, 8):
        ex = kr.createMultiThreadExecutor(streams)
        dev = _dev(data)
        outs = None
        for _ in range(4):  # plain runs, then the captured graph's
            outs = kr.runGraph(ex, mod, dev, start, T - start, outputs=outs or {})
            assert not compare_exact(_cpu(outs), want), streams
            for o in outs.values():
                o.fill_(3.0)
        # host buffers: outputs leave as their kernels end
        assert not compare_exact(kr.runGraph(ex, mod, data, start, T - start), want), streams


@pytest.mark.gpu
@pytest.mark.parametrize("key,name", [("alpha101_f32", "alpha101"), ("alpha158_f32", "alpha158")])
def test_universes_on_several_streams(key, name):
    mod = kr.Library.predefined(key).getModule(name)
    unis = [_dev(synth.ohlcv(S, T, seed=S, nan_frac=0.01)) for S, T in [(5, 90), (700, 260), (33, 310), (2049, 64)]]
    want = [_cpu(kr.runGraph(kr.createSingleThreadExecutor(), mod, u, 0, len(u["close"]))) for u in unis]
    ex = kr.createMultiThreadExecutor(8)
    for _ in range(2):
        got = kr.runGraphBatch(ex, mod, unis)
        for g, w in zip(got, want):
            assert not compare_exact(_cpu(g), w)
