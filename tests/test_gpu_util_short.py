"""aggregrate of few rows, whose blocks find the groups themselves, around the
number of rows where they stop doing so."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from oracle import utils as U
from tests.parity import compare_exact


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("T", [1, 2, 31, 32, 33, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("S", [1, 128, 300])
def test_aggregrate_of_few_rows(dt, T, S):
    rng = np.random.default_rng(T)
    xs = [rng.standard_normal((T, S)).astype(dt) for _ in range(5)]
    xs[1][rng.random((T, S)) < 0.1] = np.nan
    labels = [np.zeros(T), np.arange(T), rng.random(T) < 0.1, np.arange(T) // 31, np.arange(T) >= T - 1]
    labels = [lab.astype(dt) for lab in labels]
    labels[3][T // 2] = np.nan
    want = [U.aggregrate(x, lab) for x, lab in zip(xs, labels)]
    got = [{k: np.empty(v.shape, dt) for k, v in w.items()} for w in want]
    kr.aggregrate(kr.createSingleThreadExecutor(), xs, labels, got)
    for g, w in zip(got, want):
        assert not compare_exact(g, w)
