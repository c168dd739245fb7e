"""aggregrate's groups against its row tiles (32 rows) and corrWith's blocks
against their row lengths: the sizes where a tile, a warp or a block ends."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from oracle import utils as U
from tests.parity import compare_exact


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("T,S,sizes", [(1, 1, [1]), (70, 3, [1, 30, 1, 1, 31, 6]), (64, 129, [32, 32]),
                                       (97, 5, [33, 31, 33]), (1100, 7, [1100]), (1100, 40, [1] * 1100),
                                       (2100, 128, [9, 1024, 1, 7, 1059])])
def test_aggregrate_group_edges(dt, T, S, sizes):
    rng = np.random.default_rng(T + S)
    xs = [rng.standard_normal((T, S)).astype(dt) for _ in range(2)]
    xs[1][rng.random((T, S)) < 0.05] = np.nan
    first = np.repeat(np.arange(len(sizes)) % 7, sizes).astype(dt)
    # the second input has other labels, where a NaN label equals nothing
    second = np.repeat(np.arange((T + 4) // 5), 5)[:T].astype(dt)
    second[T // 2] = np.nan
    ex = kr.createSingleThreadExecutor()
    want = [U.aggregrate(x, lab) for x, lab in zip(xs, (first, second))]
    got = [{k: np.empty(v.shape, dt) for k, v in w.items()} for w in want]
    kr.aggregrate(ex, xs, [first, second], got)
    for g, w in zip(got, want):
        assert not compare_exact(g, w)


@pytest.mark.gpu
@pytest.mark.parametrize("S", [2, 31, 128, 129, 997, 4097, 8193])
@pytest.mark.parametrize("rank", [False, True])
def test_corrwith_row_lengths(S, rank):
    rng = np.random.default_rng(S)
    T = 5
    xs = [rng.standard_normal((T, S)).astype(np.float32) for _ in range(3)]
    xs[1] = np.floor(4 * xs[1]) / 4          # ties
    xs[2][3, 0] = np.nan                     # a NaN row is NaN
    y = (0.3 * xs[0] + rng.standard_normal((T, S))).astype(np.float32)
    outs = [np.empty(T, np.float32) for _ in xs]
    kr.corrWith(kr.createSingleThreadExecutor(), xs, y, outs, rank_inputs=rank)
    for x, o in zip(xs, outs):
        # two-float sums: rounding of the float result alone (and of a
        # correlation of two points, which is 1 or -1)
        np.testing.assert_allclose(o, U.corr_with(x, y, rank_inputs=rank), rtol=2e-6, atol=2e-6)
