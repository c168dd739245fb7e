"""corrWith in one launch (few inputs and rows) and in three (more): the same bits
for the same input and label, whatever stands beside them."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from tests.parity import compare_exact


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["TS", "STs"])
@pytest.mark.parametrize("S,T", [(8, 1), (1000, 255), (1000, 256), (1000, 257), (72, 700)])
def test_one_launch_and_three_agree(layout, S, T):
    import torch
    rng = np.random.default_rng(T)
    shape = (T, S) if layout == "TS" else (S // 8, T, 8)
    xs = [torch.from_numpy((100 + rng.standard_normal(shape)).astype(np.float32)).cuda() for _ in range(8)]
    y = torch.from_numpy((50 + rng.standard_normal(shape)).astype(np.float32)).cuda()
    ex = kr.createSingleThreadExecutor()

    def run(inputs):
        outs = [torch.full((T,), 3.0, device="cuda") for _ in inputs]
        kr.corrWith(ex, inputs, y, outs, layout)
        return {str(i): o.cpu().numpy() for i, o in enumerate(outs)}

    # 8, 320 and 1 inputs, on both sides of 2048 pairs
    few = run(xs)
    many = run(xs * 40)
    for i, x in enumerate(xs):
        assert not compare_exact(run([x]), {"0": few[str(i)]})
        assert not compare_exact({"0": many[str(i + 8)]}, {"0": few[str(i)]})
