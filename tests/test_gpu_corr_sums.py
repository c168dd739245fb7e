"""corrWith holds its sums as two-float values normalised at every addition, 256
threads a row.  The same sums restated on the CPU, for values whose mean is up to
1e5 times their deviation: there the sums' error is what the correlation shows."""
import numpy as np
import pytest

from kunquant_gb300 import runner as kr
from oracle import utils as U

F = np.float32
THREADS = 256


def _two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def _fast_two_sum(a, b):
    s = a + b
    return s, b - (s - a)


def _add(x, y):
    """The accurate double-word addition (Joldes, Muller, Popescu 2017)."""
    s, e = _two_sum(x[0], y[0])
    t, f = _two_sum(x[1], y[1])
    h, l = _fast_two_sum(s, e + t)
    return _fast_two_sum(h, l + f)


def _sum(hi, lo):
    """Row sums of hi + lo ([T][S]): a strided share a thread, a butterfly over
    each warp, the warps in order."""
    T, S = hi.shape
    pad = -S % THREADS
    hi, lo = (np.pad(v, ((0, 0), (0, pad))).reshape(T, -1, THREADS) for v in (hi, lo))
    acc = (np.zeros((T, THREADS), F), np.zeros((T, THREADS), F))
    for k in range(hi.shape[1]):
        acc = _add(acc, (hi[:, k], lo[:, k]))
    lane = np.arange(32)
    acc = tuple(v.reshape(T, THREADS // 32, 32) for v in acc)
    for o in (16, 8, 4, 2, 1):
        acc = _add(acc, tuple(v[:, :, lane ^ o] for v in acc))
    total = (np.zeros(T, F), np.zeros(T, F))
    for w in range(THREADS // 32):
        total = _add(total, tuple(v[:, w, 0] for v in acc))
    return total[0].astype(np.float64) + total[1]


def _restated(x, y):
    def prod(a, b):  # p + e is the product: 48 bits
        exact = a.astype(np.float64) * b
        p = exact.astype(F)
        return p, (exact - p).astype(F)
    S = x.shape[1]
    zero = np.zeros_like(x)
    mx, my = _sum(x, zero) / S, _sum(y, zero) / S
    mx2, my2, mxy = _sum(*prod(x, x)) / S, _sum(*prod(y, y)) / S, _sum(*prod(x, y)) / S
    return (mxy - mx * my) / (np.sqrt(mx2 - mx * mx) * np.sqrt(my2 - my * my))


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["TS", "STs"])
@pytest.mark.parametrize("S", [40, 997, 5000, 15000])
@pytest.mark.parametrize("ratio", [1e3, 1e4, 1e5])
def test_sums_of_values_far_from_zero(layout, S, ratio):
    if layout == "STs" and S % 8:
        pytest.skip("whole blocks of 8 stocks")
    rng = np.random.default_rng(S)
    T = 24
    n = rng.standard_normal((T, S))
    x = (ratio + n).astype(F)
    y = (ratio + 0.5 * n + rng.standard_normal((T, S))).astype(F)
    lay = (lambda a: a) if layout == "TS" else (
        lambda a: np.ascontiguousarray(a.T.reshape(S // 8, 8, T).transpose(0, 2, 1)))
    out = np.empty(T, F)
    kr.corrWith(kr.createSingleThreadExecutor(), [lay(x)], lay(y), [out], layout)
    # the result's rounding, and that of the double moments: six operations
    # on values ratio^2 times the variances, fused or not
    tol = 2.0 ** -24 + 8 * ratio * ratio * 2.0 ** -53
    assert np.abs(out - _restated(x, y)).max() <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("S", [40, 997, 5000, 8193, 15000])
@pytest.mark.parametrize("ratio", [0, 1e3, 1e5])
def test_sums_of_ranks(S, ratio):
    """The ranks' sums hold far more than the result shows; what the label's
    distance from zero leaves is the restated label sums'."""
    rng = np.random.default_rng(S + 1)
    T = 24
    n = rng.standard_normal((T, S))
    x = np.floor(8 * n).astype(F) if S < 1000 else n.astype(F)
    y = (ratio + 0.5 * n + rng.standard_normal((T, S))).astype(F)
    out = np.empty(T, F)
    kr.corrWith(kr.createSingleThreadExecutor(), [x], y, [out], rank_inputs=True)
    r = np.stack([U._rank_row(row) for row in x]).astype(np.float64)
    p = y.astype(np.float64) ** 2
    hi = p.astype(F)
    my, my2 = _sum(y, np.zeros_like(y)) / S, _sum(hi, (p - hi).astype(F)) / S
    mx, mx2, mxy = r.sum(1) / S, (r * r).sum(1) / S, (r * (y - ratio)).sum(1) / S + ratio * r.sum(1) / S
    want = (mxy - mx * my) / (np.sqrt(mx2 - mx * mx) * np.sqrt(my2 - my * my))
    # the result's rounding, that of the double moments (the label's second one
    # ratio^2 times its variance), and of sums of ratio * S / 2 in two floats
    tol = 2.0 ** -24 + 8 * ratio * ratio * 2.0 ** -53 + 8 * (ratio + 1) * 2.0 ** -46
    assert np.abs(out - want).max() <= tol
