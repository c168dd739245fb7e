"""Rank on rows that hold infinities beside values that the bucket maps by their
integer keys: one sign crowded towards zero, a spread that float does not hold,
and crowded rows that ask for the other map.  The result is an integer count
divided twice, so it is compared bit for bit."""
import numpy as np
import pytest

from kunquant_gb300 import build, runner as kr
from oracle.oracle import OracleProgram
from tests import golden_util as G
from tests.parity import compare_exact

_mods = {}


def _module(fixture):
    if fixture not in _mods:
        spec = G.load(fixture)[0]
        lib = kr.Library.load(build.build_module_library([spec], "kun_rank_" + fixture))
        _mods[fixture] = (lib, lib.getModule(spec["name"]), spec)
    return _mods[fixture][1:]


def _rows(S, rng):
    i = np.arange(S)
    n = rng.normal(size=S)
    rows = []
    for finite in (np.exp(13 + n), np.exp(13 + 1.5 * n), np.exp(2 * n), 1 + 1e-7 * n, 1 + 1e-15 * np.floor(40 * n),
                   np.exp(300 * rng.random(S)), 1e-300 * np.exp(n), np.exp(2 * n) * np.where(n > 0, 1, -1),
                   np.where(i % 2 == 0, 1e-8 * n, 1e8 * (1 + 1e-7 * n)), n):
        for sign in (1, -1):
            one, both = sign * finite, sign * finite
            one[S // 3] = np.inf
            both[rng.random(S) < 0.05] = np.inf
            both[rng.random(S) < 0.05] = -np.inf
            both[rng.random(S) < 0.02] = np.nan
            rows += [one, both, np.where(i == S // 2, -np.inf, one)]
    return np.stack(rows)


@pytest.mark.gpu
@pytest.mark.parametrize("fixture", ["rank_ties_nan", "rank029_f64"])
@pytest.mark.parametrize("S", [3, 64, 129, 801, 1000, 4097, 8193, 16384])
def test_rank_rows_with_infinities(fixture, S):
    mod, spec = _module(fixture)
    dt = np.float32 if spec["dtype"] == "float" else np.float64
    with np.errstate(over="ignore"):
        a = np.concatenate([_rows(S, np.random.default_rng(S + k)) for k in range(3)]).astype(dt)
    got = kr.runGraph(kr.createSingleThreadExecutor(), mod, {"a": a}, 0, len(a))
    bad = compare_exact(got, OracleProgram(spec).run({"a": a}))
    assert not bad, dict(list(bad.items())[:5])
