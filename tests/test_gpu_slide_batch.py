"""The sliding-moment form restarts its sums at every time tile: a universe's
results do not depend on the stocks and universes that run beside it."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from kunquant_gb300 import synth
from tests.parity import compare_exact


def _dev(data):
    import torch
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in data.items()}


def _cpu(out):
    return {k: v.cpu().numpy() for k, v in out.items()}


def _module():
    return kr.Library.predefined("alpha158_slide_f32").getModule("alpha158_slide")


@pytest.mark.gpu
@pytest.mark.parametrize("streams", [1, 8])
def test_universes_give_what_each_gives_alone(streams):
    mod = _module()
    unis = [_dev(synth.ohlcv(S, T, seed=S, nan_frac=0.01)) for S, T in [(5, 290), (700, 460), (33, 510), (2049, 264)]]
    want = [_cpu(kr.runGraph(kr.createSingleThreadExecutor(), mod, u, 0, len(u["close"]))) for u in unis]
    got = kr.runGraphBatch(kr.createMultiThreadExecutor(streams), mod, unis)
    for g, w in zip(got, want):
        assert not compare_exact(_cpu(g), w)


@pytest.mark.gpu
def test_stocks_and_days_beside_do_not_matter():
    mod = _module()
    S, T = 2500, 700
    data = synth.ohlcv(S, T, seed=3, nan_frac=0.01)
    ex = kr.createMultiThreadExecutor(8)
    want = _cpu(kr.runGraph(ex, mod, _dev(data), 0, T))
    few = _cpu(kr.runGraph(ex, mod, _dev({k: v[:, :40] for k, v in data.items()}), 0, T))
    assert not compare_exact(few, {k: np.ascontiguousarray(v[:, :40]) for k, v in want.items()})
    early = _cpu(kr.runGraph(ex, mod, _dev(data), 0, 300))
    assert not compare_exact(early, {k: v[:300] for k, v in want.items()})
