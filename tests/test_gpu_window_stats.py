"""Quantiles (interpolated in two-float arithmetic) and window regressions
(straight-line divisions) on values where their fast forms end: equal and nearly
equal neighbours, opposite signs, zeros, infinities, values out of range, NaN;
against the oracle bit for bit."""
import numpy as np
import pytest

from kunquant_gb300 import build, runner as kr
from oracle.oracle import OracleProgram
from tests.parity import compare_exact

W = 10


def _spec(name, ops, outs):
    ops = [dict({"p": -1}, **o) for o in ops]
    for k, (i, out) in enumerate(outs):
        ops.append({"k": "Output", "in": [i], "p": -1, "buf": k + 1})
    bufs = [{"id": 0, "name": "a", "kind": "INPUT", "num_users": 1, "unreliable_count": 0, "window": W + 1}]
    bufs += [{"id": k + 1, "name": out, "kind": "OUTPUT", "num_users": 0, "unreliable_count": 0, "window": 1}
             for k, (_, out) in enumerate(outs)]
    return {"name": name, "dtype": "float", "input_layout": "TS", "output_layout": "TS", "blocking_len": 8,
            "aligned": False, "options": {}, "buffers": bufs, "single_value_inputs": [],
            "stages": [{"name": name, "kind": "ts", "in": [0], "out": [b["id"] for b in bufs[1:]], "deps": [],
                        "pending": 0, "ops": ops}]}


def _quantile_spec():
    return _spec("quantile_unit",
                 [{"k": "Input", "in": [], "buf": 0}, {"k": "BackRef", "in": [0], "window": W},
                  {"k": "SkipListState", "in": [1, 0], "window": W},
                  {"k": "SkipListQuantile", "in": [2], "q": "0.2"}, {"k": "SkipListQuantile", "in": [2], "q": "0.8"},
                  {"k": "SkipListQuantile", "in": [2], "q": "0.37"}], [(3, "q20"), (4, "q80"), (5, "q37")])


def _regression_spec():
    return _spec("regression_unit",
                 [{"k": "Input", "in": [], "buf": 0}, {"k": "WindowedLinearRegression", "in": [0], "window": W},
                  {"k": "WindowedLinearRegressionRSqaureImpl", "in": [1]},
                  {"k": "WindowedLinearRegressionSlopeImpl", "in": [1]},
                  {"k": "WindowedLinearRegressionResiImpl", "in": [1, 0]}],
                 [(2, "rsq"), (3, "slope"), (4, "resi")])


def _values(T, rng):
    n = rng.standard_normal(T)
    cols = [100 + n, 1e-7 * n + 100, np.floor(3 * n), n, np.full(T, 7.5), np.where(n > 0, 1e30, -1e30) * (1 + 0.1 * n),
            1e-42 * np.floor(100 * n), np.exp(30 * n), np.where(rng.random(T) < 0.1, np.inf, n), np.zeros(T),
            np.where(rng.random(T) < 0.2, np.nan, 50 + n), np.where(n > 0, 0.1 * (1 + 1e-7 * n), -0.1),
            np.arange(T) * 0.5, np.where(np.arange(T) < T // 2, 3.0, 3.0 + 1e-6 * np.arange(T))]
    return np.stack(cols, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_quantile_spec, _regression_spec])
@pytest.mark.parametrize("T", [1, 9, 11, 63, 700])
def test_window_statistics_at_the_ends_of_their_range(make, T):
    spec = make()
    lib = kr.Library.load(build.build_module_library([spec], "kun_" + spec["name"]))
    with np.errstate(over="ignore"):
        a = np.concatenate([_values(T, np.random.default_rng(k)) for k in range(6)], 1).astype(np.float32)
    got = kr.runGraph(kr.createSingleThreadExecutor(), lib.getModule(spec["name"]), {"a": a}, 0, T)
    bad = compare_exact(got, OracleProgram(spec).run({"a": a}))
    assert not bad, bad
