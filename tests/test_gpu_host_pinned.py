"""Runs on the caller's own pinned memory, alone and mixed with pageable and device
buffers, repeated, on both sides of the sizes where their copies change."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from kunquant_gb300 import synth
from kunquant_gb300.graph import predefined_spec
from oracle.oracle import OracleProgram
from tests.parity import compare_exact


def _pinned(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


# KB a buffer of 163: 1, 65, 190, 195, 480 (73 MB)
@pytest.mark.gpu
@pytest.mark.parametrize("S,T", [(3, 70), (64, 260), (152, 320), (156, 320), (300, 400)])
@pytest.mark.parametrize("streams", [1, 8])
def test_pinned_and_mixed_host_runs(S, T, streams):
    mod = kr.Library.predefined("alpha158_f32").getModule("alpha158")
    prog = OracleProgram(predefined_spec("alpha158_f32"))
    ex = kr.createMultiThreadExecutor(streams)
    names = sorted(mod.getOutputNames())
    keep = {k: _pinned(np.zeros((T, S), np.float32)) for k in names}
    for seed in range(4):
        data = synth.ohlcv(S, T, seed=seed, nan_frac=0.01)
        want = prog.run(data)
        # all pinned; pinned inputs; pinned outputs; every other buffer
        every = [lambda i: True, lambda i: False, lambda i: True, lambda i: i % 2 == 0][seed]
        inputs = {k: _pinned(v) if seed < 2 or i % 2 else v for i, (k, v) in enumerate(data.items())}
        outs = {k: keep[k] if every(i) else np.empty((T, S), np.float32) for i, k in enumerate(names)}
        for _ in range(2):
            for o in outs.values():
                o[:] = 3
            got = kr.runGraph(ex, mod, inputs, 0, T, outputs=outs)
            assert not compare_exact(got, want), seed
