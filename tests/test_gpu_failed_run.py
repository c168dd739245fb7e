"""A run whose Rank rows are too long fails at that stage's launch, after kernels
of earlier stages have been queued: it waits for them, so that the caller's
buffers are its own again and the executor's next run is a clean one."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from kunquant_gb300 import synth
from tests.parity import compare_exact

LONG = 16385  # one stock above Rank's longest row


def _dev(data):
    import torch
    return {k: torch.from_numpy(v).cuda() for k, v in data.items()}


def _host(o):
    return o.copy() if isinstance(o, np.ndarray) else o.cpu().numpy()


def _cpu(out):
    return {k: _host(v) for k, v in out.items()}


@pytest.mark.gpu
@pytest.mark.parametrize("streams", [1, 8])
@pytest.mark.parametrize("where", ["device", "host", "batch"])
def test_a_failed_run_leaves_nothing_behind(streams, where):
    import torch
    mod = kr.Library.predefined("alpha101_f32").getModule("alpha101")
    good = _dev(synth.ohlcv(300, 90, seed=1, nan_frac=0.01))
    want = _cpu(kr.runGraph(kr.createSingleThreadExecutor(), mod, good, 0, 90))
    bad = synth.ohlcv(LONG, 70, seed=2)
    ex = kr.createMultiThreadExecutor(streams)
    for _ in range(3):  # plain, and where a repeated run would be captured
        with pytest.raises(kr.KunError, match="launch failed|grouped Rank failed"):
            if where == "device":
                inputs = _dev(bad)
                outs = {k: torch.full((70, LONG), 3.0, device="cuda") for k in mod.getOutputNames()}
                kr.runGraph(ex, mod, inputs, 0, 70, outputs=outs)
            elif where == "host":
                outs = {k: np.full((70, LONG), 3.0, np.float32) for k in mod.getOutputNames()}
                kr.runGraph(ex, mod, bad, 0, 70, outputs=outs)
            else:
                inputs = [good, _dev(bad)]
                kr.runGraphBatch(ex, mod, inputs)
        if where != "batch":
            # nothing writes to the caller's outputs any more
            before = {k: _host(o) for k, o in outs.items()}
            torch.cuda.synchronize()
            after = {k: _host(o) for k, o in outs.items()}
            assert not compare_exact(after, before)
        assert not compare_exact(_cpu(kr.runGraph(ex, mod, good, 0, 90)), want)
